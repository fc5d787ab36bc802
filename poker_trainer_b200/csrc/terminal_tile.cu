// Tile-per-block terminal evaluation: T terminals of one board at a time, the
// fixed-point prefix sums of warp_terminal_task (warp_terminal.cuh) with the T
// terminals' prefixes side by side, [position][T].
//
// One terminal at a time, every hand's six prefixes are random 8-byte reads
// of shared memory, four wavefronts and more for a warp's 32, and every index
// and conversion is spent on one terminal: about 136 warp instructions and 58
// wavefronts per 32 (hand, terminal) pairs (terminal_group.cu). Here a thread
// works on two terminals of a tile and reads both with one 16-byte access; T / 2
// threads read a whole row of the tile, 8 T contiguous bytes, whatever hand it
// belongs to. An index is read once for T terminals, an entry of a reach row
// is converted once (not once per list that holds it), and what remains is
// about 50 instructions and 33 wavefronts per 32 pairs.
//
// A tile of live terminals (dead subtrees are skipped when it is formed),
// all showdowns or all folds:
//   A  each row's maximum is known: entries become fixed point, written at
//      their hand's place in the strength order (X);
//   B  runs of X are summed; then, while one warp scans those sums and one
//      forms the next tile, each card's list is gathered from X into exclusive
//      prefixes of its own, 0 first and the card's total last;
//   C  X becomes its exclusive prefixes in place, and the next tile's rows are
//      requested;
//   D  every hand's values from eight rows of the tile.
// Values are bit-identical to the other kernels': the same integer sums, the
// same conversions and the same rounding order per terminal kind.
//
// Bound by shared memory's latency and barriers at one block an SM: 0.53 of its
// one wavefront a cycle on a flop, 0.46 with sampled cards (ncu; short scoreboard
// and barrier are the largest stalls). A tile of 16
// terminals at 470 hands takes 14,600 cycles, of which maxima 360, X 1530, run
// sums 870, card lists 3040, placing 1850 and values 6940 (two warps per
// terminal: 16 x 1125 cycles). A flop's terminals, ms a traversal: 10.8 to 8.3.
// 24 warps (80 registers, spills) take 10.6 ms; forming half of X by integer
// shifts, or reading the next hand while one is formed, 8.9.
#include <cuda_runtime.h>

#include <cstdint>

#include "pdl.cuh"
#include "plan.hpp"
#include "warp_terminal.cuh"

namespace dcfr {

constexpr int TILE_WARPS = 16;
constexpr int TILE_STEPS = 2;  // row loads (float4 of two terminals) per thread
constexpr int TILE_RUN = 8;    // X entries per thread in the strength scan

// One terminal of a tile.
struct TileTask {
  uint32_t slot, row, frow, scalar;
  double a, b, c, d;
};

struct TileSmem {
  size_t rows, wsum, task, max, list, spos, clist, rec, same, seg, total;
  __host__ __device__ TileSmem(int T, int n_o, int n_p) {
    auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    rows = 0;
    wsum = rows + (size_t)(3 * n_o + 53) * T * 8;
    task = wsum + (size_t)(TILE_WARPS + 1) * T * 8;
    max = task + 2 * (size_t)T * sizeof(TileTask);
    list = up16(max + 2 * (size_t)T * 4 + 16);
    spos = up16(list + TILE_THREADS * 2);
    clist = up16(spos + ((size_t)n_o + 8) * 2);
    rec = up16(clist + (size_t)2 * n_o * 2);
    same = up16(rec + (size_t)n_p * 16);
    seg = up16(same + (size_t)n_p * 2);
    total = up16(seg + FAST_SEGS * 2);
  }
};

__device__ __forceinline__ longlong2 operator+(longlong2 a, longlong2 b) { return make_longlong2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ longlong2 operator-(longlong2 a, longlong2 b) { return make_longlong2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ longlong2 shfl_up2(longlong2 v, int d) {
  return make_longlong2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}

// Jobs are runs of at most TILE_THREADS tasks on one layout and of one class
// (TermUnit::pad), largest first. Blocks claim them from a counter that the
// traversal's start has cleared: the share of live tasks varies from job to
// job by more than static ranges even out (a flop with sampled cards: 0.79 ms
// a traversal against 0.52). A block claims its next job while it works on
// one.
template <int T>
__global__ void __launch_bounds__(TILE_THREADS, 1)
    tile_terminal_kernel(FastArgs A, const FastTask* __restrict__ tasks, const TermUnit* __restrict__ jobs, int njobs,
                         uint32_t* __restrict__ counter, int n_o_max, int n_p_max) {
  extern __shared__ __align__(16) unsigned char smem_t[];
  constexpr int TP = T / 2;             // threads across a row of the tile
  constexpr int WPW = 32 / TP;          // rows a warp reads at once
  constexpr int NW = TILE_WARPS * WPW;  // walkers: rows the block reads at once
  constexpr int HU = T / 8;             // consecutive hands a walker evaluates (32-byte stores across a warp)
  const TileSmem L_(T, n_o_max, n_p_max);
  longlong2* G = reinterpret_cast<longlong2*>(smem_t + L_.rows);  // row r: G[r * TP + tp]
  longlong2* wsum = reinterpret_cast<longlong2*>(smem_t + L_.wsum);
  TileTask* stask = reinterpret_cast<TileTask*>(smem_t + L_.task);  // [2][T]
  uint32_t* smax = reinterpret_cast<uint32_t*>(smem_t + L_.max);    // [2][T]
  uint16_t* slist = reinterpret_cast<uint16_t*>(smem_t + L_.list);
  uint16_t* spos = reinterpret_cast<uint16_t*>(smem_t + L_.spos);
  uint16_t* clist = reinterpret_cast<uint16_t*>(smem_t + L_.clist);
  uint4* srec = reinterpret_cast<uint4*>(smem_t + L_.rec);
  uint16_t* ssame = reinterpret_cast<uint16_t*>(smem_t + L_.same);
  uint16_t* sseg = reinterpret_cast<uint16_t*>(smem_t + L_.seg);
  __shared__ uint32_t swin[TILE_WARPS];
  __shared__ int s_job;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tp = lane % TP, walker = warp * WPW + lane / TP;
  const int p = A.p, o = p ^ 1;
  const int hpo = o ? A.hp[1] : A.hp[0], hpp = p ? A.hp[1] : A.hp[0], np = p ? A.n[1] : A.n[0];
  // A job's layout. The card lists hold places in the strength order, and a
  // layout position pos of card c's segment is row pos + 1 + c (every list has
  // one row more than hands).
  int n = 0;
  auto stage = [&](uint32_t layout) {
    const size_t lay = (size_t)layout * 2 + p;
    const uint16_t* gseg = A.seg + lay * FAST_SEGS;
    const uint16_t* gcat = A.cat + lay * A.cstride;
    const uint4* grec = A.rec + lay * A.tstride;
    const int L = gseg[FAST_SEGS - 1];
    n = gseg[1];
    if (tid < FAST_SEGS) sseg[tid] = gseg[tid];
    for (int j = tid; j < hpo; j += TILE_THREADS) spos[j] = 0xFFFF;
    __syncthreads();
    for (int k = tid; k < n; k += TILE_THREADS) spos[gcat[k]] = (uint16_t)k;
    __syncthreads();
    for (int k = n + tid; k < L; k += TILE_THREADS) clist[k - n] = spos[gcat[k]];
    for (int h = tid; h < np; h += TILE_THREADS) {
      const uint4 q = grec[h];
      const uint32_t a = q.w & 0xFFu, b = (q.w >> 8) & 0xFFu;
      const uint32_t ta = sseg[2 + a] + 1u + a, tb = sseg[2 + b] + 1u + b;
      const uint32_t da = (1u + a) * 0x10001u, db = (1u + b) * 0x10001u;
      // Not on the board: no showdown value (w = 0xFFFF).
      srec[h] = (q.w >> 16) ? make_uint4(q.x, q.y + da, q.z + db, ta | tb << 16)
                            : make_uint4(0xFFFFu, 0u, 0u, ta | tb << 16);
      const uint32_t sm = A.same[h];
      ssame[h] = sm == NONE32 ? (uint16_t)0xFFFF : spos[sm];
    }
    __syncthreads();
  };
  // The live tasks among the TILE_THREADS from `from` on, in order: their
  // places go to slist, their number is returned.
  auto window = [&](int from, int end) {
    const int i = from + tid;
    const bool live = i < end && A.alive[tasks[i].slot] != 0;  // dead subtree (cfr.rs:267-274): rows untouched
    const uint32_t m = __ballot_sync(0xffffffffu, live);
    if (lane == 0) swin[warp] = __popc(m);
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < TILE_WARPS; w++) {
      const uint32_t c = swin[w];
      if (w < warp) before += c;
      total += c;
    }
    if (live) slist[before + __popc(m & ((1u << lane) - 1u))] = (uint16_t)tid;
    __syncthreads();
    return (int)total;
  };
  // Warp 15: the tile of live tasks [at, at + T) of the window from `from` on.
  auto form = [&](int from, int at, int live, int buf) {
    if (lane < T && at + lane < live) {
      const FastTask k = tasks[from + slist[at + lane]];
      stask[buf * T + lane] = TileTask{k.slot, k.row, k.frow,
                                       k.kind == T_FOLD_SCALAR || k.kind == T_SHOWDOWN_SCALAR ? 1u : 0u,
                                       k.a, k.b, k.c, k.d};
      // The row is requested a phase later: into L2 by then.
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A.reach + (size_t)k.slot * A.stride),
                   "r"(hpo * 4));
    }
  };
  // The tile's rows: this thread's two terminals, hands j..j+3 of each step. A
  // warp reads WPW * 16 contiguous bytes of each row.
  float4 r0[TILE_STEPS], r1[TILE_STEPS];
  auto hand = [&](int s) { return ((s * TILE_WARPS + warp) * WPW + lane / TP) * 4; };
  auto request = [&](int buf, int count) {
    const bool on0 = 2 * tp < count, on1 = 2 * tp + 1 < count;
    const float* a = A.reach + (size_t)(on0 ? stask[buf * T + 2 * tp].slot : 0u) * A.stride;
    const float* b = A.reach + (size_t)(on1 ? stask[buf * T + 2 * tp + 1].slot : 0u) * A.stride;
#pragma unroll
    for (int s = 0; s < TILE_STEPS; s++) {
      const int j = hand(s);
      r0[s] = on0 && j < hpo ? *reinterpret_cast<const float4*>(a + j) : make_float4(0.f, 0.f, 0.f, 0.f);
      r1[s] = on1 && j < hpo ? *reinterpret_cast<const float4*>(b + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto publish_max = [&](int buf) {
    float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
    for (int s = 0; s < TILE_STEPS; s++) {
      m0 = fmaxf(m0, fmaxf(fmaxf(r0[s].x, r0[s].y), fmaxf(r0[s].z, r0[s].w)));
      m1 = fmaxf(m1, fmaxf(fmaxf(r1[s].x, r1[s].y), fmaxf(r1[s].z, r1[s].w)));
    }
#pragma unroll
    for (int d = TP; d < 32; d <<= 1) {
      m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, d));
      m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, d));
    }
    if (lane < TP) {
      atomicMax(smax + buf * T + 2 * lane, __float_as_uint(m0));
      atomicMax(smax + buf * T + 2 * lane + 1, __float_as_uint(m1));
    }
  };
  if (tid < 2 * T) smax[tid] = 0u;
  int job = blockIdx.x;  // the first gridDim.x jobs are the blocks' first
  if (job >= njobs) return;
  uint32_t staged = jobs[job].layout;
  stage(staged);
  pdl_wait();
  pdl_trigger();
  int buf = 0;
  while (job < njobs) {
    const TermUnit U = jobs[job];
    __syncthreads();
    if (tid == 0) s_job = (int)(gridDim.x + atomicAdd(counter, 1u));
    if (U.layout != staged) {
      staged = U.layout;
      stage(staged);
    }
    const bool fold = U.pad == TILE_FOLD;
    const int from = (int)U.first;
    const int live = window(from, from + (int)U.count);
    if (warp == TILE_WARPS - 1) form(from, 0, live, buf);
    __syncthreads();
    request(buf, min(T, live));
    for (int tile = 0; tile < live; tile += T) {
      const int count = min(T, live - tile);
      publish_max(buf);
      __syncthreads();  // (A) row maxima; the previous tile is read
      {
        const double s0 = pow2(scale_exponent(__uint_as_float(smax[buf * T + 2 * tp])));
        const double s1 = pow2(scale_exponent(__uint_as_float(smax[buf * T + 2 * tp + 1])));
#pragma unroll
        for (int s = 0; s < TILE_STEPS; s++) {
          const int j = hand(s);
          if (j >= hpo) break;
          const ushort4 to = *reinterpret_cast<const ushort4*>(spos + j);
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const uint32_t row = (&to.x)[k];
            if (row != 0xFFFFu) G[row * TP + tp] = make_longlong2(fixed((&r0[s].x)[k], s0), fixed((&r1[s].x)[k], s1));
          }
        }
      }
      __syncthreads();  // (B) X is written
      const int E = (n + NW - 1) / NW;
      const int x0 = walker * E, x1 = min(n, x0 + E);
      longlong2 x[TILE_RUN], run = make_longlong2(0, 0);
#pragma unroll
      for (int i = 0; i < TILE_RUN; i++) {
        x[i] = x0 + i < x1 ? G[(x0 + i) * TP + tp] : make_longlong2(0, 0);
        run = run + x[i];
      }
      longlong2 inc = run;
#pragma unroll
      for (int d = TP; d < 32; d <<= 1) {
        const longlong2 y = shfl_up2(inc, d);
        if (lane >= d) inc = inc + y;
      }
      if (lane >= 32 - TP) wsum[warp * TP + tp] = inc;
      __syncthreads();
      // Each card's list, a walker a card: exclusive prefixes (folds: the total).
      if (walker < 52) {
        const int c = walker, k0 = sseg[1 + c] - n, k1 = sseg[2 + c] - n;
        longlong2* to = G + (size_t)(sseg[1 + c] + 1 + c) * TP + tp;
        longlong2 acc = make_longlong2(0, 0);
        int k = k0;
        for (; k + 4 <= k1; k += 4) {
          longlong2 v[4];
#pragma unroll
          for (int i = 0; i < 4; i++) v[i] = G[(int)clist[k + i] * TP + tp];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            if (!fold) to[(k - k0 + i) * TP] = acc;
            acc = acc + v[i];
          }
        }
        for (; k < k1; k++) {
          const longlong2 v = G[(int)clist[k] * TP + tp];
          if (!fold) to[(k - k0) * TP] = acc;
          acc = acc + v;
        }
        to[(k1 - k0) * TP] = acc;
      }
      if (warp == TILE_WARPS - 2 && lane < TP) {
        // The warps' runs: sums of the warps before, and the total last.
        longlong2 before = make_longlong2(0, 0);
        for (int w = 0; w < TILE_WARPS; w++) {
          const longlong2 y = wsum[w * TP + lane];
          wsum[w * TP + lane] = before;
          before = before + y;
        }
        wsum[TILE_WARPS * TP + lane] = before;
      }
      if (warp == TILE_WARPS - 1) form(from, tile + T, live, buf ^ 1);
      __syncthreads();  // (C) runs and cards are summed, X is gathered
      const longlong2 T0 = wsum[TILE_WARPS * TP + tp];
      longlong2 acc = wsum[warp * TP + tp] + inc - run;
      if (!fold) {
#pragma unroll
        for (int i = 0; i < TILE_RUN; i++)
          if (x0 + i < x1) {
            G[(x0 + i) * TP + tp] = acc;
            acc = acc + x[i];
          }
        if (tid < TP) G[n * TP + tp] = T0;
      }
      // This thread's two terminals, and the next tile's rows.
      const TileTask Ta = stask[buf * T + 2 * tp], Tb = stask[buf * T + 2 * tp + 1];
      const double i0 = pow2(-scale_exponent(__uint_as_float(smax[buf * T + 2 * tp])));
      const double i1 = pow2(-scale_exponent(__uint_as_float(smax[buf * T + 2 * tp + 1])));
      const bool on0 = 2 * tp < count, on1 = 2 * tp + 1 < count;
      request(buf ^ 1, min(T, live - tile - T));
      __syncthreads();  // (D) prefixes are written
      if (tid < T) smax[buf * T + tid] = 0u;
      float* out0 = A.vals + (size_t)(on0 ? Ta.row : 0u) * A.stride;
      float* out1 = A.vals + (size_t)(on1 ? Tb.row : 0u) * A.stride;
      const double pa0 = Ta.a * i0, pa1 = Tb.a * i1, pb0 = Ta.b * i0, pb1 = Tb.b * i1;
      auto at = [&](uint32_t row) { return G[row * TP + tp]; };
      auto put = [&](float* to, int h, const float (&v)[HU]) {
        if constexpr (HU == 2) *reinterpret_cast<float2*>(to + h) = make_float2(v[0], v[1]);
        else to[h] = v[0];
      };
      if (U.pad == TILE_PLAIN) {
        for (int h = walker * HU; h < hpp; h += NW * HU) {
          float v0[HU], v1[HU];
#pragma unroll
          for (int e = 0; e < HU; e++) {
            v0[e] = v1[e] = 0.0f;
            if (h + e >= np) continue;
            const uint4 q = srec[h + e];
            if ((q.x & 0xFFFFu) == 0xFFFFu) continue;
            const longlong2 W = at(q.x & 0xFFFFu) - at(q.y & 0xFFFFu) - at(q.z & 0xFFFFu);
            const longlong2 Lx = T0 - at(q.x >> 16) + at(q.y >> 16) + at(q.z >> 16) - at(q.w & 0xFFFFu) - at(q.w >> 16);
            double x0 = pa0 * (double)W.x, x1 = pa1 * (double)W.y;
            x0 += pb0 * (double)Lx.x;
            x1 += pb1 * (double)Lx.y;
            v0[e] = (float)x0;
            v1[e] = (float)x1;
          }
          if (on0) put(out0, h, v0);
          if (on1) put(out1, h, v1);
        }
      } else {
        const double pc0 = Ta.c * i0, pc1 = Tb.c * i1, pd0 = Ta.d * i0, pd1 = Tb.d * i1;
        const bool f0 = on0 && Ta.frow != NONE32, f1 = on1 && Tb.frow != NONE32;
        float* fo0 = A.vals + (size_t)(f0 ? Ta.frow : 0u) * A.stride;
        float* fo1 = A.vals + (size_t)(f1 ? Tb.frow : 0u) * A.stride;
        for (int h = walker * HU; h < hpp; h += NW * HU) {
          float v0[HU], v1[HU], g0[HU], g1[HU];
#pragma unroll
          for (int e = 0; e < HU; e++) {
            v0[e] = v1[e] = g0[e] = g1[e] = 0.0f;
            if (h + e >= np) continue;
            const uint4 q = srec[h + e];
            const uint32_t sm = ssame[h + e];
            const longlong2 ta = at(q.w & 0xFFFFu), tb = at(q.w >> 16);
            longlong2 si = make_longlong2(0, 0);
            if (sm != 0xFFFFu) si = fold ? at(sm) : at(sm + 1) - at(sm);
            const longlong2 F = T0 - ta - tb + si;
            if (fold) {
              v0[e] = (Ta.scalar && T0.x == 0) ? 0.0f : (float)(pa0 * (double)F.x);
              v1[e] = (Tb.scalar && T0.y == 0) ? 0.0f : (float)(pa1 * (double)F.y);
              continue;
            }
            if ((q.x & 0xFFFFu) != 0xFFFFu) {
              const longlong2 Gw = at(q.x & 0xFFFFu), Gs = at(q.x >> 16);
              const longlong2 aw = at(q.y & 0xFFFFu), as = at(q.y >> 16), bw = at(q.z & 0xFFFFu), bs = at(q.z >> 16);
              const longlong2 W = Gw - aw - bw, Lx = T0 - Gs + as + bs - ta - tb;
              const longlong2 eq = (Gs - Gw) - (as - aw) - (bs - bw) + si;
              auto value = [&](const TileTask& K, double pa, double pb, double pc, long long w, long long l,
                               long long q2) {
                float v;
                if (K.scalar) {
                  v = (float)(pa * (double)w) + (float)(pb * (double)l);
                } else {
                  double res = pa * (double)w;
                  res += pb * (double)l;
                  v = (float)res;
                }
                if (K.c != 0.0) v += (float)(pc * (double)q2);
                return v;
              };
              v0[e] = value(Ta, pa0, pb0, pc0, W.x, Lx.x, eq.x);
              v1[e] = value(Tb, pa1, pb1, pc1, W.y, Lx.y, eq.y);
            }
            if (f0) g0[e] = (float)(pd0 * (double)F.x);
            if (f1) g1[e] = (float)(pd1 * (double)F.y);
          }
          if (on0) put(out0, h, v0);
          if (on1) put(out1, h, v1);
          if (f0) put(fo0, h, g0);
          if (f1) put(fo1, h, g1);
        }
      }
      buf ^= 1;
    }
    job = s_job;
  }
}

// Terminals per tile for hand lists of up to n[0], n[1]: the widest that fits
// shared memory and the threads' registers; 0: none.
int tile_terminal_setup(int n0, int n1, int hp0, int hp1) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 0;
  const int n = n0 > n1 ? n0 : n1, hp = hp0 > hp1 ? hp0 : hp1;
  for (int T : {16, 8}) {
    const void* fn = T == 16 ? (const void*)tile_terminal_kernel<16> : (const void*)tile_terminal_kernel<8>;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return 0;
    const int limit = optin - (int)fa.sharedSizeBytes;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) return 0;
    const int walkers = TILE_WARPS * 64 / T;
    if (TileSmem(T, hp, n).total <= (size_t)limit && (n + walkers - 1) / walkers <= TILE_RUN &&
        hp <= TILE_STEPS * TILE_WARPS * (64 / T) * 4)
      return T;
  }
  return 0;
}

void launch_tile_terminal(const FastArgs& A, const FastTask* tasks, const TermUnit* jobs, int njobs, uint32_t* counter,
                          int T, int max_blocks, cudaStream_t s) {
  if (njobs <= 0) return;
  const int blocks = njobs < max_blocks ? njobs : max_blocks;
  const int n = A.n[0] > A.n[1] ? A.n[0] : A.n[1], hp = A.hp[0] > A.hp[1] ? A.hp[0] : A.hp[1];
  launch_dependent(T == 16 ? tile_terminal_kernel<16> : tile_terminal_kernel<8>, dim3((unsigned)blocks), TILE_THREADS,
                   TileSmem(T, hp, n).total, s, A, tasks, jobs, njobs, counter, hp, n);
}

}  // namespace dcfr
