// Terminal values in exact precision: fold and showdown evaluation with exact
// card removal, bit-identical to the reference's evaluators
// (AhanDatta/Poker-Trainer crates/solver/src/eval.rs:40-379).
//
// A block takes one terminal. What must be sequential for the CPU's rounding
// is no more than the sums themselves: the running sum over the strength order
// (upwards for the win part and the paired fold, downwards for the lose part)
// and each card's sum over the hands that hold it, 2 + 104 independent chains
// of f64 additions over the scan layout's segments (fast_layout_kernel: the
// hands by strength, then by card and strength; folds: in hand order). Every
// chain leaves its partial sums in place, and each hand reads the ones at its
// own strength, where the reference's sweep emits it.
//
// Bound by the latency of the chain over all hands (1081 dependent f64
// additions) where there are few terminals, by the chains' shared-memory
// traffic where there are many. Against a warp walking the merged strength
// lists of up to 32 terminals, one step per hand of either player (a
// traversal's launches, ms): river, 29 terminals of 1081 hands, 0.457 to
// 0.018; turn, 11,678 of about 800 hands, 0.716 to 0.204, of 470 hands 0.360 to
// 0.128; flop with sampled cards, 50,964, 2.235 to 0.591.
#include <cuda_runtime.h>

#include <cstdint>

#include "pdl.cuh"
#include "plan.hpp"

namespace dcfr {

constexpr int EXACT_THREADS = 256;
struct ExactSmem {
  size_t up, down, row, cat, seg, total;
  __host__ __device__ ExactSmem(int stride, int cstride, int tstride) {
    auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    up = 0;
    down = up + (size_t)cstride * 8;
    row = down + (size_t)cstride * 8;
    cat = up16(row + (size_t)stride * 4);
    seg = up16(cat + (size_t)cstride * 2);
    total = up16(seg + FAST_SEGS * 2);
  }
};

// In-place running sums of x[k0..k1), upwards or downwards.
template <bool UP>
__device__ __forceinline__ void chain(double* x, int k0, int k1) {
  double s = 0.0;
  constexpr int B = 8;
  int k = 0;
  const int n = k1 - k0;
  double* base = UP ? x + k0 : x + k1 - 1;
  constexpr int d = UP ? 1 : -1;
  for (; k + B <= n; k += B) {
    double v[B];
#pragma unroll
    for (int i = 0; i < B; i++) v[i] = base[d * (k + i)];
#pragma unroll
    for (int i = 0; i < B; i++) {
      s += v[i];
      base[d * (k + i)] = s;
    }
  }
  for (; k < n; k++) {
    s += base[d * k];
    base[d * k] = s;
  }
}

__global__ void __launch_bounds__(EXACT_THREADS) exact_terminal_kernel(FastArgs A, const FastTask* __restrict__ tasks,
                                                                       int ntasks, uint32_t fold_layout) {
  extern __shared__ __align__(16) unsigned char smem_x[];
  const ExactSmem L_(A.stride, A.cstride, A.tstride);
  double* up = reinterpret_cast<double*>(smem_x + L_.up);
  double* down = reinterpret_cast<double*>(smem_x + L_.down);
  float* row = reinterpret_cast<float*>(smem_x + L_.row);
  uint16_t* cat = reinterpret_cast<uint16_t*>(smem_x + L_.cat);
  uint16_t* seg = reinterpret_cast<uint16_t*>(smem_x + L_.seg);
  const int p = A.p, o = p ^ 1, tid = threadIdx.x;
  const int hpo = o ? A.hp[1] : A.hp[0], hpp = p ? A.hp[1] : A.hp[0], np = p ? A.n[1] : A.n[0];
  pdl_wait();
  pdl_trigger();
  turn_pass(A.turn);
  uint32_t staged = NONE32;
  int L = 0;
  for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
    const FastTask T = tasks[t];
    if (A.alive[T.slot] == 0) continue;  // dead subtree: rows untouched
    const bool fold = T.kind == T_FOLD_SCALAR || T.kind == T_FOLD_BATCH;
    const bool scalar = T.kind == T_FOLD_SCALAR || T.kind == T_SHOWDOWN_SCALAR;
    const uint32_t layout = fold ? fold_layout : T.board;
    const size_t lay = (size_t)layout * 2 + p;
    __syncthreads();  // the previous terminal is done with shared memory
    for (int i = tid; i < hpo / 4; i += EXACT_THREADS)
      reinterpret_cast<float4*>(row)[i] = reinterpret_cast<const float4*>(A.reach + (size_t)T.slot * A.stride)[i];
    if (layout != staged) {
      const uint16_t* gseg = A.seg + lay * FAST_SEGS;
      if (tid < FAST_SEGS) seg[tid] = gseg[tid];
      L = gseg[FAST_SEGS - 1];
      const uint16_t* gcat = A.cat + lay * A.cstride;
      for (int k = tid; k < L; k += EXACT_THREADS) cat[k] = gcat[k];
      staged = layout;
    }
    __syncthreads();
    for (int k = tid; k < L; k += EXACT_THREADS) {
      const double x = (double)row[cat[k]];
      up[k] = x;
      down[k] = x;
    }
    __syncthreads();
    // The chains: one warp each for the two long ones, the cards' on others.
    if (tid == 0) chain<true>(up, 0, seg[1]);
    else if (tid >= 64 && tid < 64 + 52) chain<true>(up, seg[1 + tid - 64], seg[2 + tid - 64]);
    if (!fold) {
      if (tid == 32) chain<false>(down, 0, seg[1]);
      else if (tid >= 128 && tid < 128 + 52) chain<false>(down, seg[1 + tid - 128], seg[2 + tid - 128]);
    }
    __syncthreads();
    auto below = [&](int k, int k0) { return k == k0 ? 0.0 : up[k - 1]; };   // sum of [k0, k)
    auto above = [&](int k, int k1) { return k == k1 ? 0.0 : down[k]; };     // sum of [k, k1), from the top
    const int ct = seg[1];
    const double total = below(ct, 0);
    float* out = A.vals + (size_t)T.row * A.stride;
    float* fout = T.frow != NONE32 ? A.vals + (size_t)T.frow * A.stride : nullptr;
    const uint4* rec = A.rec + lay * A.tstride;
    for (int h = tid; h < hpp; h += EXACT_THREADS) {
      float v = 0.0f, fv = 0.0f;
      if (h < np) {
        const uint4 q = rec[h];
        const int a = (int)(q.w & 0xFF), b = (int)((q.w >> 8) & 0xFF);
        const int a0 = seg[1 + a], a1 = seg[2 + a], b0 = seg[1 + b], b1 = seg[2 + b];
        const uint32_t sm = A.same[h];
        const double s = sm == NONE32 ? 0.0 : (double)row[sm];
        const double ta = below(a1, a0), tb = below(b1, b0);
        if (fold) {
          // eval_fold (eval.rs:55-63), fold_batch (eval.rs:197-205).
          if (scalar) v = total == 0.0 ? 0.0f : (float)(T.a * ((total - (ta + tb)) + s));
          else v = (float)(T.a * (((total - ta) - tb) + s));
        } else {
          if (q.w >> 16) {
            const int w = (int)(q.x & 0xFFFF), e = (int)(q.x >> 16);
            const int aw = (int)(q.y & 0xFFFF), ae = (int)(q.y >> 16), bw = (int)(q.z & 0xFFFF), be = (int)(q.z >> 16);
            const double S = below(w, 0), va = below(aw, a0), vb = below(bw, b0);
            const double D = above(e, ct), da = above(ae, a1), db = above(be, b1);
            if (scalar) {
              v = (float)(T.a * (S - (va + vb))) + (float)(T.b * (D - (da + db)));
            } else {
              const double win = T.a * ((S - va) - vb), lose = T.b * ((D - da) - db);
              v = (float)(win + lose);
            }
            if (T.c != 0.0) {
              // add_ties (eval.rs:347-379): sums over the hands of equal
              // strength, and those of them holding each card, from zero.
              double eq = 0.0, ea = 0.0, eb = 0.0;
              for (int k = w; k < e; k++) eq += (double)row[cat[k]];
              for (int k = aw; k < ae; k++) ea += (double)row[cat[k]];
              for (int k = bw; k < be; k++) eb += (double)row[cat[k]];
              v += (float)(T.c * ((eq - (ea + eb)) + s));
            }
          }
          // The paired fold of showdown_batch (eval.rs:292-300).
          if (fout) fv = (float)(T.d * (((total - ta) - tb) + s));
        }
      }
      out[h] = v;
      if (fout) fout[h] = fv;
    }
  }
}

// Blocks per SM of exact_terminal_kernel; 0 if its shared memory does not fit.
int exact_terminal_setup(int stride, int cstride, int tstride) {
  int dev = 0, optin = 0, blocks = 0;
  const size_t smem = ExactSmem(stride, cstride, tstride).total;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      smem > (size_t)optin ||
      cudaFuncSetAttribute(exact_terminal_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, exact_terminal_kernel, EXACT_THREADS, smem) != cudaSuccess)
    return 0;
  return blocks;
}

void launch_exact_terminal(const FastArgs& A, const FastTask* tasks, int ntasks, uint32_t fold_layout, int max_blocks,
                           cudaStream_t s) {
  if (ntasks <= 0) return;
  const int blocks = ntasks < max_blocks ? ntasks : max_blocks;
  launch_dependent(exact_terminal_kernel, (unsigned)blocks, EXACT_THREADS,
                   ExactSmem(A.stride, A.cstride, A.tstride).total, s, A, tasks, ntasks, fold_layout);
}

}  // namespace dcfr
