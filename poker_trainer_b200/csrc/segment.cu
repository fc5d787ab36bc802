// The decision nodes of the street segment that no chance node precedes (a
// traversal's root segment) in one launch per direction, and the up pass of
// one traversal together with the down pass of the next, whose opponent is
// the player that the up pass has just updated.
//
// Everything these passes compute is per hand, so a block takes one slice of
// SEG_SLICE hands, one a lane, through every node of the segment: its warps
// share a level's nodes and meet at a block barrier between levels, with no
// launch and no other block in between. Everything the slice needs is fetched
// at once by cp.async: the storage rows before the wait on the previous grid
// (no kernel between two segment passes touches them), the value rows and
// liveness flags after it. The levels then run at shared-memory latency, and
// the down pass finds the regrets that the up pass has just updated.
//
// Bound by the latency of a node's own instruction stream (a warp alone on
// its scheduler), hence one hand a lane: with 4 hands a lane, as the level
// kernels have, a pass took 9.0 us on average where it takes 7.1 (16 decision
// nodes, 1081 hands), and the fetches one after another in place of all at
// once cost 3 us of a pass. One launch per level took 2.5 us a level for the
// same work: a river iteration of 1081 hands went from 52 us (19 launches) to
// 22.5 us (6 launches), one of 260 hands from 38 to 15.3 us, a turn's root
// street from 20 to 11 us a traversal.
//
// What couples the slices is the dead-subtree rule (cfr.rs:267-274): a node
// is skipped only if NO opponent hand reaches it, and a slice sees its own
// hands alone. Where a slice's hands do not reach a node, it writes zeros to
// the children's rows and defers the node's strategy sums, whose update a
// live node needs whether its hands are reached or not; the up pass of the
// same traversal, a later launch that sees every slice's liveness flags,
// makes up for it before anything else.
#include <cuda_runtime.h>

#include <cstdint>

#include "engine.hpp"
#include "pdl.cuh"
#include "plan.hpp"
#include "row_items.cuh"
#include "segment.cuh"

namespace dcfr {

constexpr int SEG_WARPS = 8;

// Shared memory: the slice's rows (storage of the player both passes update,
// the up pass's value rows, the down pass's reach rows), both passes' plan
// records, liveness flags and deferred flags.
struct SegSmem {
  size_t reg, sum, val, reach, up, down, ulive, dlive, deferred, total;
  __host__ __device__ explicit SegSmem(const SegPass& P) {
    auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const size_t row = SEG_SLICE * 4;
    reg = 0;
    sum = reg + P.n_rows * row;
    val = sum + P.n_rows * row;
    reach = val + P.U.n_rows * row;
    up = reach + P.D.n_slots * row;
    down = up + P.U.bytes;
    ulive = down + (P.D.bytes - P.D.o_down);
    dlive = up16(ulive + (size_t)P.U.n_slots * 4);
    deferred = up16(dlive + (size_t)P.D.n_slots * 4);
    total = up16(deferred + P.U.n_down);
  }
};

size_t segment_smem(const SegPass& P) { return SegSmem(P).total; }

__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_landed() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

__device__ __forceinline__ void stage(unsigned char* dst, const unsigned char* src, uint32_t bytes) {
  for (uint32_t i = threadIdx.x * 16; i < bytes; i += blockDim.x * 16) copy16(dst + i, src + i);
}

template <int MODE, int MAXA>
__global__ void __launch_bounds__(SEG_WARPS * 32, 2) segment_kernel(const __grid_constant__ SegPass P) {
  extern __shared__ __align__(16) unsigned char smem_s[];
  const SegSmem L(P);
  float* reg = reinterpret_cast<float*>(smem_s + L.reg);
  float* sum = reinterpret_cast<float*>(smem_s + L.sum);
  float* val = reinterpret_cast<float*>(smem_s + L.val);
  float* rch = reinterpret_cast<float*>(smem_s + L.reach);
  const SegUp* ut = reinterpret_cast<const SegUp*>(smem_s + L.up);
  const SegDown* ft = reinterpret_cast<const SegDown*>(smem_s + L.up + P.U.o_down);
  const SegRow* vl = reinterpret_cast<const SegRow*>(smem_s + L.up + P.U.o_vals);
  const uint32_t* us = reinterpret_cast<const uint32_t*>(smem_s + L.up + P.U.o_slots);
  const uint32_t* ulevs = reinterpret_cast<const uint32_t*>(smem_s + L.up + P.U.o_levs);
  const SegDown* dt = reinterpret_cast<const SegDown*>(smem_s + L.down);
  const uint32_t* ds = reinterpret_cast<const uint32_t*>(smem_s + L.down + (P.D.o_slots - P.D.o_down));
  const uint32_t* dlevs =
      reinterpret_cast<const uint32_t*>(smem_s + L.down + (P.D.o_levs - P.D.o_down)) + P.D.nup + 1;
  uint32_t* ulive = reinterpret_cast<uint32_t*>(smem_s + L.ulive);
  uint32_t* dlive = reinterpret_cast<uint32_t*>(smem_s + L.dlive);
  uint8_t* deferred = smem_s + L.deferred;
  const int sl = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = sl * SEG_SLICE + lane;
  const bool do_up = P.U.blob != nullptr, do_down = P.D.blob != nullptr;
  // The player both passes update: the up pass's traverser, the down pass's
  // opponent.
  const RowArgs& AQ = do_up ? P.up : P.down;
  const int q = do_up ? AQ.p : AQ.p ^ 1;
  const int hp = pick(q, AQ.hp), hpo = pick(q ^ 1, AQ.hp), stride = AQ.stride;
  const bool valid = h < hp;
  pdl_trigger();
  // Before the wait: plan data, and what no kernel since the last segment
  // pass but one has touched (every kernel lets the next start only when all
  // before it are complete, or at its own start if it is a segment pass, and
  // no two segment passes follow one another).
  if (do_up) stage(smem_s + L.up, P.U.blob, P.U.bytes);
  if (do_down) stage(smem_s + L.down, P.D.blob + P.D.o_down, P.D.bytes - P.D.o_down);
  const bool want_sums = do_down || MODE == M_AVG;
  for (uint32_t k0 = warp; k0 < P.n_rows; k0 += SEG_WARPS * 32) {
    // A warp's rows: one load of their offsets, then all their copies.
    const uint32_t mine = k0 + (uint32_t)lane * SEG_WARPS;
    const unsigned long long at = mine < P.n_rows ? P.rows[mine] : 0ull;
    for (int j = 0; j < 32 && k0 + (uint32_t)j * SEG_WARPS < P.n_rows; j++) {
      const uint32_t k = k0 + (uint32_t)j * SEG_WARPS;
      const unsigned long long off = __shfl_sync(0xffffffffu, at, j);
      if (valid) {
        if (MODE == M_CFR) copy4(reg + k * SEG_SLICE + lane, AQ.regrets + off + h);
        if (want_sums) copy4(sum + k * SEG_SLICE + lane, AQ.sums + off + h);
      } else {
        reg[k * SEG_SLICE + lane] = 0.0f;
        sum[k * SEG_SLICE + lane] = 0.0f;
      }
    }
  }
  if (MODE == M_CFR && do_up)
    for (uint32_t i = tid; i < P.U.n_down; i += blockDim.x) deferred[i] = P.up_deferred[(size_t)sl * P.U.n_down + i];
  if (do_down)
    for (uint32_t i = tid; i < P.D.n_slots; i += blockDim.x) dlive[i] = 0;
  const float root = do_down && h < stride ? P.roots[h] : 0.0f;
  copies_landed();
  pdl_wait();
  if (do_up) {
    for (uint32_t i = warp; i < P.U.n_vals; i += SEG_WARPS) {
      const SegRow R = vl[i];
      if (h < stride) copy4(val + R.row * SEG_SLICE + lane, P.up.vals + (size_t)R.node * stride + h);
      else val[R.row * SEG_SLICE + lane] = 0.0f;
    }
    for (uint32_t i = tid; i < P.U.n_slots; i += blockDim.x) ulive[i] = P.up.alive[us[i]];
  }
  if (do_down && warp == 0) {
    rch[lane] = root;
    if (h < stride) P.down.reach[(size_t)ds[0] * stride + h] = root;
    const bool some = __any_sync(0xffffffffu, valid && root != 0.0f);
    if (lane == 0) {
      dlive[0] = some ? 1u : 0u;
      if (sl == 0) P.down.alive[ds[0]] = 1u;
    }
  }
  DiscountD d{}, dd{};  // the up pass's and the down pass's
  if (MODE == M_CFR) {
    d = *AQ.disc;
    dd = do_down ? *P.down.disc : d;
  }
  copies_landed();
  if (do_up) {
    if (MODE == M_CFR) {
      // The deferred strategy sums of nodes that turned out live: this
      // slice's hands have no reach there.
      for (uint32_t b = warp * 32; b < P.U.n_down; b += SEG_WARPS * 32) {
        const uint32_t i = b + lane;
        uint32_t m = __ballot_sync(0xffffffffu, i < P.U.n_down && deferred[i] != 0 && ulive[ft[i].in_slot] != 0);
        for (; m; m &= m - 1) {
          const SegDown& T = ft[b + __ffs(m) - 1];
          if (h >= hpo) continue;
          float x[MAXA];
#pragma unroll
          for (int a = 0; a < MAXA; a++)
            x[a] = P.up.regrets[T.gstore + (size_t)min(a, (int)T.nchild - 1) * hpo + h];
          to_strategy<MAXA, true>(x, (int)T.nchild, T.uniform);
#pragma unroll
          for (int a = 0; a < MAXA; a++)
            if (a < (int)T.nchild) {
              float* s = P.up.sums + T.gstore + (size_t)a * hpo + h;
              *s = next_sum(*s, x[a], 0.0f, d);
            }
        }
      }
    }
    for (uint32_t l = 0; l < P.U.nup; l++) {
      const uint32_t e = ulevs[l + 1];
      for (uint32_t i = ulevs[l] + warp; i < e; i += SEG_WARPS) {
        const SegUp T = ut[i];
        if (ulive[T.slot] == 0) continue;  // dead subtree
        const int na = (int)T.nchild;
        // An action past the node's last reads the last one's row and is
        // left out of every sum: no branch per action.
        float v[MAXA], out = 0.0f;
#pragma unroll
        for (int a = 0; a < MAXA; a++) v[a] = val[(T.child + min(a, na - 1)) * SEG_SLICE + lane];
        if (T.kind == U_OPP_SUM) {
          // Opponent node (cfr.rs:421-432).
          bool on[MAXA];
#pragma unroll
          for (int a = 0; a < MAXA; a++) on[a] = a < na && ulive[T.child_slot + min(a, na - 1)] != 0;
#pragma unroll
          for (int a = 0; a < MAXA; a++) out = on[a] ? out + v[a] : out;
        } else if (MODE == M_BR) {
          out = v[0];
#pragma unroll
          for (int a = 1; a < MAXA; a++) out = v[a] > out ? v[a] : out;
        } else if (MODE == M_AVG) {
          float x[MAXA];
#pragma unroll
          for (int a = 0; a < MAXA; a++) x[a] = sum[(T.store + min(a, na - 1)) * SEG_SLICE + lane];
          to_strategy<MAXA, false>(x, na, T.uniform);
#pragma unroll
          for (int a = 0; a < MAXA; a++) out = a < na ? out + x[a] * v[a] : out;
        } else {
          // own_node_update (cfr.rs:315-382).
          float r[MAXA];
#pragma unroll
          for (int a = 0; a < MAXA; a++) r[a] = reg[(T.store + min(a, na - 1)) * SEG_SLICE + lane];
          own_value<MAXA>(r, v, na, T.uniform, out);
          float* to = P.up.regrets + T.gstore + h;
#pragma unroll
          for (int a = 0; a < MAXA; a++) {
            const float x = next_regret(r[a], v[a], out, d);
            if (a < na) {
              reg[(T.store + a) * SEG_SLICE + lane] = x;
              if (valid) to[(size_t)a * hp] = x;
            }
          }
        }
        val[T.node * SEG_SLICE + lane] = out;
        if (valid) P.up.vals[(size_t)T.gnode * stride + h] = out;
      }
      __syncthreads();
    }
    if (P.root_out && warp == 0 && h < stride)
      P.root_out[h] = valid ? val[lane] : P.up.vals[(size_t)P.U.root * stride + h];
  }
  if (do_down) {
    const float* from = MODE == M_CFR ? reg : sum;
    for (uint32_t l = 0; l < P.D.ndown; l++) {
      const uint32_t e = dlevs[l + 1];
      for (uint32_t i = dlevs[l] + warp; i < e; i += SEG_WARPS) {
        const SegDown T = dt[i];
        const int na = (int)T.nchild;
        const bool some = dlive[T.in_slot] != 0;
        float* to = P.down.reach + (size_t)T.gslot * stride + h;
        if (some) {
          const float r = rch[T.in_slot * SEG_SLICE + lane];
          float x[MAXA], s[MAXA];
#pragma unroll
          for (int a = 0; a < MAXA; a++) {
            x[a] = from[(T.store + min(a, na - 1)) * SEG_SLICE + lane];
            s[a] = MODE == M_CFR ? sum[(T.store + min(a, na - 1)) * SEG_SLICE + lane] : 0.0f;
          }
          to_strategy<MAXA, MODE == M_CFR>(x, na, T.uniform);
          uint32_t kids = 0;
#pragma unroll
          for (int a = 0; a < MAXA; a++) {
            const float c = x[a] * r;
            kids |= (__any_sync(0xffffffffu, valid && c != 0.0f) ? 1u : 0u) << a;
            if (a < na) {
              rch[(T.out_slot + a) * SEG_SLICE + lane] = c;
              if (valid) {
                to[(size_t)a * stride] = c;
                if (MODE == M_CFR) P.down.sums[T.gstore + (size_t)a * hp + h] = next_sum(s[a], x[a], r, dd);
              }
            }
          }
          if (lane < na && (kids >> lane & 1u)) {
            dlive[T.out_slot + lane] = 1u;
            P.down.alive[T.gslot + lane] = 1u;
          }
        } else if (valid) {
          for (int a = 0; a < na; a++) to[(size_t)a * stride] = 0.0f;
        }
        if (MODE == M_CFR && lane == 0) P.down_deferred[(size_t)sl * P.D.n_down + i] = some ? 0 : 1;
      }
      __syncthreads();
    }
  }
}

template <int MODE>
static const void* segment_fn(int maxa) {
  if (maxa <= 4) return (const void*)segment_kernel<MODE, 4>;
  if (maxa <= 8) return (const void*)segment_kernel<MODE, 8>;
  return (const void*)segment_kernel<MODE, MAX_ACTIONS>;
}
static const void* segment_fn(int mode, int maxa) {
  return mode == M_CFR ? segment_fn<M_CFR>(maxa) : mode == M_BR ? segment_fn<M_BR>(maxa) : segment_fn<M_AVG>(maxa);
}

cudaError_t segment_setup() {
  for (int mode : {M_CFR, M_BR, M_AVG})
    for (int maxa : {4, 8, MAX_ACTIONS}) {
      const cudaError_t e =
          cudaFuncSetAttribute(segment_fn(mode, maxa), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEG_SMEM_MAX);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

void launch_segment(int mode, int maxa, const SegPass& P, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)P.slices);
  cfg.blockDim = dim3(SEG_WARPS * 32);
  cfg.dynamicSmemBytes = segment_smem(P);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* params[] = {(void*)&P};
  cudaLaunchKernelExC(&cfg, segment_fn(mode, maxa), params);
}

}  // namespace dcfr
