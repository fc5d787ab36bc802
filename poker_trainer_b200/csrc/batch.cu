// Batched river solves: hundreds of independent river subgames of uneven tree
// size solved together, launched from captured CUDA graphs.
//
// Every spot is a complete river game (its own board, ranges, pot, stacks
// and bet menu) built by the same host code as a single solve (game.cpp), so
// its tree, storage order and arithmetic are those of the reference solver
// (crates/solver/src/tree.rs, cfr.rs, river.rs, eval.rs). The spots share one
// numbering of reach slots, rows (each spot's as long as its own longer range; a
// traversal writes its opponent's hands, and past them a reach row may hold the
// other traversal's) and terminal tasks, and an iteration is four launches
// over all of them: for each traversal a row pass and the terminals, the up
// pass of a traversal being one launch with the down pass of the next.
//   * Row passes (batch_row_kernel): everything is per hand, so a slice of 32
//     or 64 hands of a spot goes through all its nodes on its own, taking each
//     node's rows from global memory; a slice's part in the dead-subtree
//     rule is deferred as in segment.cu.
//   * Terminals: the single solve's kernels over all spots' tasks, a unit of
//     the scan layouts per spot (terminal_group.cu; terminal_fast.cu for few).
// A persistent block per spot, for whole iterations, left a spot's 400 nodes
// to 6 warps and the GPU to its longest spots: 37 spots of 1081 hands took
// 1622 us an iteration where they now take 105, 512 spots 2078 us, now 960.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <numeric>
#include <vector>

#include "batch.hpp"
#include "pdl.cuh"
#include "row_items.cuh"
#include "segment.cuh"
#include "warp_terminal.cuh"

namespace dcfr {

namespace {

// One traversal's part of a spot: its tasks in one array for all spots, levels
// [levs[lev + l], levs[lev + l + 1]) (up: deepest first).
struct BatchPart {
  uint32_t up_lev, nup, down_lev, ndown;
};
struct SpotD {
  uint32_t slot;    // reach slot 0 of the spot (its root's)
  uint32_t nslots;  // slots of its larger traversal
  uint32_t reach;   // reach row of slot 0, and value row of the root (ROW_UNITs)
  uint32_t vals;
  int32_t stride;   // entries of its rows
  uint32_t pad;
  int32_t hp[2];
  BatchPart part[2];
};

// A block's work: a spot, and its slice or the first of its warps' slices.
struct RowItem {
  uint32_t spot, slice;
};

// SegUp / SegDown (plan.hpp) with slots counted from the spot's first, and rows
// (node, child, gnode; gslot: the first child's reach row) in ROW_UNITs.
struct BatchPass {
  const SpotD* spots;
  const RowItem* items;
  int stride;               // of roots and root_out
  int max_up, max_fix, max_down, max_slots;  // largest spot: records staged, slots
  uint32_t n_fix, n_down;   // down tasks of the up and of the down traversal
  float* regrets;
  float* sums;
  float* reach;
  float* vals;
  uint32_t* alive[2];       // per traverser
  const DiscountD* disc;       // the up pass's
  const DiscountD* down_disc;
  int up_p, down_p;         // traversers of the two passes, -1: not wanted
  const SegUp* up;
  const SegDown* fix;       // the up traversal's down tasks
  const uint32_t* up_levs;
  uint8_t* up_deferred;     // [slices][down task]
  const SegDown* down;
  const uint32_t* down_levs;
  uint8_t* down_deferred;
  const float* roots;       // [spot][traverser][stride]
  float* root_out;          // likewise, or null
};

// A block works on one spot: 8 warps on one slice of it, a level's nodes side
// by side with a barrier between levels (SHARE), or 4 warps on a slice each,
// every warp taking the nodes one after another.
template <bool SHARE>
struct RowShape {
  static constexpr int WARPS = SHARE ? 8 : 4;
  static constexpr int SLICES = SHARE ? 1 : WARPS;
  static constexpr int V = SHARE ? 1 : 2;  // hands a lane
  static constexpr int SLICE = 32 * V;     // hands a slice
};

// A lane's V hands of a row, by one load or store.
template <int V>
struct Row {
  float x[V];
  __device__ __forceinline__ static Row load(const float* p) {
    Row r;
    if constexpr (V == 1) r.x[0] = *p;
    else {
      const float2 t = *reinterpret_cast<const float2*>(p);
      r.x[0] = t.x;
      r.x[1] = t.y;
    }
    return r;
  }
  __device__ __forceinline__ void store(float* p) const {
    if constexpr (V == 1) *p = x[0];
    else *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  }
};

struct RowSmem {
  size_t up, fix, down, live, any, total;
  __host__ __device__ RowSmem(int max_up, int max_fix, int max_down, int max_slots, int slices) {
    up = 0;
    fix = up + (size_t)max_up * sizeof(SegUp);
    down = fix + (size_t)max_fix * sizeof(SegDown);
    live = down + (size_t)max_down * sizeof(SegDown);
    any = live + (size_t)max_slots;
    total = any + (size_t)slices * max_slots;
  }
};

template <typename T>
__device__ __forceinline__ void stage_records(T* dst, const T* src, uint32_t count) {
  for (uint32_t i = threadIdx.x; i < count * (uint32_t)(sizeof(T) / 16); i += blockDim.x)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(reinterpret_cast<uint4*>(dst) + i)),
                 "l"(reinterpret_cast<const uint4*>(src) + i)
                 : "memory");
}

// Bound by the latency of a node's loads (value rows, then the next node's),
// so the plan records and liveness flags are in shared memory, no load waits
// for another, a lane has two hands where that leaves enough slices, and as
// many warps run as the registers allow without spills (512 spots, us an
// iteration: two hands a lane 28 warps an SM 1193 with spills, 24 warps 1057,
// 20 warps 1018, 16 warps 1021; four hands 12 warps 1038, 16 warps 1080; one
// hand 28 warps 1140). A node's work is by its own number of actions, not the
// batch's largest: 37 spots of up to 8 actions 126 to 113.
// STAGED: shared memory holds the plan records of the batch's largest spot; a
// larger one's are read where they are (trees of 8,000 nodes and more).
template <int MODE, int MAXA, bool SHARE, bool STAGED>
__global__ void __launch_bounds__(RowShape<SHARE>::WARPS * 32, SHARE ? 3 : 5)
    batch_row_kernel(const __grid_constant__ BatchPass P) {
  extern __shared__ __align__(16) unsigned char smem_b[];
  using R = Row<RowShape<SHARE>::V>;
  constexpr int W = RowShape<SHARE>::WARPS, GS = RowShape<SHARE>::SLICES, V = RowShape<SHARE>::V;
  const RowSmem L(P.max_up, P.max_fix, P.max_down, P.max_slots, GS);
  uint8_t* live = smem_b + L.live;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t* any = smem_b + L.any + (SHARE ? 0 : (size_t)warp * P.max_slots);
  pdl_trigger();
  const RowItem item = P.items[blockIdx.x];
  const uint32_t sp = item.spot;
  const int sl = (int)item.slice + (SHARE ? 0 : warp);
  const int w0 = SHARE ? warp : 0;
  constexpr int WS = SHARE ? W : 1;
  const SpotD S = P.spots[sp];
  const int h = sl * RowShape<SHARE>::SLICE + lane * V;  // the lane's first; hand counts are padded to eights
  const size_t stride = (size_t)S.stride;
  const bool do_up = P.up_p >= 0, do_down = P.down_p >= 0;
  const BatchPart U = pick(do_up ? P.up_p : 0, S.part), D = pick(do_down ? P.down_p : 0, S.part);
  uint32_t u0 = 0, un = 0, f0 = 0, fn = 0, d0 = 0, dn = 0;
  if (do_up) {
    u0 = P.up_levs[U.up_lev];
    un = P.up_levs[U.up_lev + U.nup] - u0;
    if constexpr (STAGED) stage_records(reinterpret_cast<SegUp*>(smem_b + L.up), P.up + u0, un);
    if (MODE == M_CFR) {
      f0 = P.up_levs[U.down_lev];
      fn = P.up_levs[U.down_lev + U.ndown] - f0;
      if constexpr (STAGED) stage_records(reinterpret_cast<SegDown*>(smem_b + L.fix), P.fix + f0, fn);
    }
  }
  if (do_down) {
    d0 = P.down_levs[D.down_lev];
    dn = P.down_levs[D.down_lev + D.ndown] - d0;
    if constexpr (STAGED) stage_records(reinterpret_cast<SegDown*>(smem_b + L.down), P.down + d0, dn);
  }
  const SegUp* const ut = STAGED ? reinterpret_cast<const SegUp*>(smem_b + L.up) : P.up + u0;
  const SegDown* const ft = STAGED ? reinterpret_cast<const SegDown*>(smem_b + L.fix) : P.fix + f0;
  const SegDown* const dt = STAGED ? reinterpret_cast<const SegDown*>(smem_b + L.down) : P.down + d0;
  for (uint32_t i = threadIdx.x; i < S.nslots * GS; i += W * 32)
    smem_b[L.any + (i / S.nslots) * P.max_slots + i % S.nslots] = 0;
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  pdl_wait();
  DiscountD d{}, dd{};  // the up pass's and the down pass's
  if (MODE == M_CFR) {
    d = *P.disc;
    dd = *P.down_disc;
  }
  if (do_up)
    for (uint32_t i = threadIdx.x; i < S.nslots; i += W * 32) live[i] = pick(P.up_p, P.alive)[S.slot + i] != 0;
  __syncthreads();
  if (!SHARE && sl * RowShape<SHARE>::SLICE >= S.stride) return;
  if (do_up) {
    const int hp = pick(P.up_p, S.hp), hpo = pick(P.up_p ^ 1, S.hp);
    if (MODE == M_CFR) {
      // The deferred strategy sums of nodes that turned out live.
      for (uint32_t b = w0 * 32; b < fn; b += WS * 32) {
        const uint32_t i = b + lane;
        uint32_t m = __ballot_sync(0xffffffffu, i < fn && P.up_deferred[(size_t)sl * P.n_fix + f0 + i] != 0 &&
                                                    live[ft[i].in_slot] != 0);
        for (; m; m &= m - 1) {
          const SegDown& T = ft[b + __ffs(m) - 1];
          if (h >= hpo) continue;
          by_actions<MAXA>((int)T.nchild, [&](auto most, int na) {
            constexpr int M = decltype(most)::value;
            float x[V][M];
#pragma unroll
            for (int a = 0; a < M; a++) {
              const R v = a < na ? R::load(P.regrets + T.gstore + (size_t)a * hpo + h) : R{};
#pragma unroll
              for (int j = 0; j < V; j++) x[j][a] = v.x[j];
            }
#pragma unroll
            for (int j = 0; j < V; j++) to_strategy<M, true>(x[j], na, T.uniform);
#pragma unroll
            for (int a = 0; a < M; a++)
              if (a < na) {
                float* at = P.sums + T.gstore + (size_t)a * hpo + h;
                R q = R::load(at);
#pragma unroll
                for (int j = 0; j < V; j++) q.x[j] = next_sum(q.x[j], x[j][a], 0.0f, d);
                q.store(at);
              }
          });
        }
      }
    }
    for (uint32_t l = 0; l < (SHARE ? U.nup : 1u); l++) {
      // Not shared: all tasks in one go, in order.
      const uint32_t e = SHARE ? P.up_levs[U.up_lev + l + 1] - u0 : un;
      for (uint32_t i = (SHARE ? P.up_levs[U.up_lev + l] - u0 : 0u) + w0; i < e; i += WS) {
        const SegUp& T = ut[i];
        if (live[T.slot] == 0 || h >= hp) continue;  // dead subtree
        const float* vp = P.vals + (size_t)T.child * ROW_UNIT + h;
        R out{};
        by_actions<MAXA>((int)T.nchild, [&](auto most, int na) {
          constexpr int M = decltype(most)::value;
          R v[M];
          if (T.kind == U_OPP_SUM) {
#pragma unroll
            for (int a = 0; a < M; a++)
              if (a < na) v[a] = R::load(vp + (size_t)a * stride);
#pragma unroll
            for (int a = 0; a < M; a++)
              if (a < na && live[T.child_slot + a] != 0)
#pragma unroll
                for (int j = 0; j < V; j++) out.x[j] += v[a].x[j];
          } else if (MODE == M_BR) {
#pragma unroll
            for (int a = 0; a < M; a++)
              if (a < na) v[a] = R::load(vp + (size_t)a * stride);
            out = v[0];
#pragma unroll
            for (int a = 1; a < M; a++)
              if (a < na)
#pragma unroll
                for (int j = 0; j < V; j++) out.x[j] = v[a].x[j] > out.x[j] ? v[a].x[j] : out.x[j];
          } else {
            float* to = (MODE == M_CFR ? P.regrets : P.sums) + T.gstore + h;
            float c[V][M], r[V][M];  // child values; regrets or sums
#pragma unroll
            for (int a = 0; a < M; a++) {
              const R x = a < na ? R::load(vp + (size_t)a * stride) : R{};
              const R y = a < na ? R::load(to + (size_t)a * hp) : R{};
#pragma unroll
              for (int j = 0; j < V; j++) {
                c[j][a] = x.x[j];
                r[j][a] = y.x[j];
              }
            }
            if (MODE == M_AVG) {
#pragma unroll
              for (int j = 0; j < V; j++) {
                to_strategy<M, false>(r[j], na, T.uniform);
#pragma unroll
                for (int a = 0; a < M; a++) out.x[j] = a < na ? out.x[j] + r[j][a] * c[j][a] : out.x[j];
              }
            } else {
#pragma unroll
              for (int j = 0; j < V; j++) own_value<M>(r[j], c[j], na, T.uniform, out.x[j]);
#pragma unroll
              for (int a = 0; a < M; a++)
                if (a < na) {
                  R q;
#pragma unroll
                  for (int j = 0; j < V; j++) q.x[j] = next_regret(r[j][a], c[j][a], out.x[j], d);
                  q.store(to + (size_t)a * hp);
                }
            }
          }
        });
        out.store(P.vals + (size_t)T.gnode * ROW_UNIT + h);
      }
      if (SHARE) __syncthreads();
    }
    if (P.root_out && w0 == 0 && h < S.stride)
      R::load(P.vals + (size_t)S.vals * ROW_UNIT + h).store(P.root_out + ((size_t)sp * 2 + P.up_p) * P.stride + h);
  }
  if (do_down) {
    uint32_t* alive = pick(P.down_p, P.alive) + S.slot;
    const int hp = pick(P.down_p ^ 1, S.hp);
    const bool valid = h < hp;
    if (w0 == 0) {
      const R r = h < S.stride ? R::load(P.roots + ((size_t)sp * 2 + P.down_p) * P.stride + h) : R{};
      if (h < S.stride) r.store(P.reach + (size_t)S.reach * ROW_UNIT + h);
      bool some = false;
#pragma unroll
      for (int j = 0; j < V; j++) some |= valid && r.x[j] != 0.0f;
      some = __any_sync(0xffffffffu, some);
      if (lane == 0) {
        any[0] = some ? 1 : 0;
        if (sl == 0) alive[0] = 1u;
      }
    }
    if (SHARE) __syncthreads();
    else __syncwarp();
    for (uint32_t l = 0; l < (SHARE ? D.ndown : 1u); l++) {
      const uint32_t e = SHARE ? P.down_levs[D.down_lev + l + 1] - d0 : dn;
      for (uint32_t i = (SHARE ? P.down_levs[D.down_lev + l] - d0 : 0u) + w0; i < e; i += WS) {
        const SegDown& T = dt[i];
        const int na = (int)T.nchild;
        const bool some = any[T.in_slot] != 0;
        float* to = P.reach + (size_t)T.gslot * ROW_UNIT + h;
        if (some) {
          const R r = valid ? R::load(P.reach + (size_t)S.reach * ROW_UNIT + T.in_slot * stride + h) : R{};
          const float* from = (MODE == M_CFR ? P.regrets : P.sums) + T.gstore + h;
          float* sums = P.sums + T.gstore + h;
          uint32_t kids = 0;  // children that a hand of the lane reaches
          by_actions<MAXA>(na, [&](auto most, int na) {
            constexpr int M = decltype(most)::value;
            float x[V][M];
            R s[M];
#pragma unroll
            for (int a = 0; a < M; a++) {
              const R v = a < na && valid ? R::load(from + (size_t)a * hp) : R{};
              s[a] = MODE == M_CFR && a < na && valid ? R::load(sums + (size_t)a * hp) : R{};
#pragma unroll
              for (int j = 0; j < V; j++) x[j][a] = v.x[j];
            }
#pragma unroll
            for (int j = 0; j < V; j++) to_strategy<M, MODE == M_CFR>(x[j], na, T.uniform);
#pragma unroll
            for (int a = 0; a < M; a++)
              if (a < na && valid) {
                R c;
#pragma unroll
                for (int j = 0; j < V; j++) {
                  c.x[j] = x[j][a] * r.x[j];
                  kids |= c.x[j] != 0.0f ? 1u << a : 0u;
                  if (MODE == M_CFR) s[a].x[j] = next_sum(s[a].x[j], x[j][a], r.x[j], dd);
                }
                c.store(to + (size_t)a * stride);
                if (MODE == M_CFR) s[a].store(sums + (size_t)a * hp);
              }
          });
          kids = __reduce_or_sync(0xffffffffu, kids);
          if (kids >> lane & 1u) {
            any[T.out_slot + lane] = 1;
            alive[T.out_slot + lane] = 1u;
          }
        } else if (valid) {
          for (int a = 0; a < na; a++) R{}.store(to + (size_t)a * stride);
        }
        if (MODE == M_CFR && lane == 0) P.down_deferred[(size_t)sl * P.n_down + d0 + i] = some ? 0 : 1;
        if (!SHARE) __syncwarp();
      }
      if (SHARE) __syncthreads();
    }
  }
}

template <int MODE, bool SHARE>
const void* row_fn(int maxa, bool staged) {
  if (!staged) return (const void*)batch_row_kernel<MODE, MAX_ACTIONS, SHARE, false>;
  if (maxa <= 4) return (const void*)batch_row_kernel<MODE, 4, SHARE, true>;
  if (maxa <= 8) return (const void*)batch_row_kernel<MODE, 8, SHARE, true>;
  return (const void*)batch_row_kernel<MODE, MAX_ACTIONS, SHARE, true>;
}
template <bool SHARE>
const void* row_fn(int mode, int maxa, bool staged) {
  return mode == M_CFR  ? row_fn<M_CFR, SHARE>(maxa, staged)
         : mode == M_BR ? row_fn<M_BR, SHARE>(maxa, staged)
                        : row_fn<M_AVG, SHARE>(maxa, staged);
}

// What dcfr_batch_tuning::warps is accepted up to: shared memory for that many
// terminals, one a warp, on the largest spot. (The kernels take no more
// terminals a block than fit them, whatever is set: Impl::max_groups.)
size_t tuning_smem(int stride, int cstride, int tstride, int max_slots, int warps) {
  auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
  const size_t fixed = up16((size_t)max_slots * 4) + up16(sizeof(DiscountD)) + 16 + up16((size_t)stride * 2) +
                       up16((size_t)cstride * 2) + up16((size_t)tstride * 16) + up16(FAST_SEGS * 2);
  return fixed + (size_t)warps * (up16((size_t)stride * 4) + up16(warp_prefix_entries(cstride) * 8));
}

Status cuda_st(cudaError_t e, const char* what) { return cuda_status(e, what); }

#define BK(call)                                  \
  do {                                            \
    Status _s = cuda_st((call), #call);           \
    if (!_s.ok()) return _s;                      \
  } while (0)

template <class T>
Status balloc(T*& p, size_t count, const char* what) {
  p = nullptr;
  if (count == 0) count = 1;
  cudaError_t e = cudaMalloc((void**)&p, count * sizeof(T));
  if (e != cudaSuccess) {
    Status s = cuda_status(e, what);
    s.msg += " (" + std::to_string(count * sizeof(T)) + " bytes)";
    return s;
  }
  return Status();
}

template <class T>
void bfree(T*& p) {
  if (p) cudaFree(p);
  p = nullptr;
}

template <class T>
Status upload(T*& d, const std::vector<T>& h, const char* what) {
  Status s = balloc(d, h.size(), what);
  if (!s.ok()) return s;
  if (h.empty()) return Status();
  BK(cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
  BK(cudaStreamSynchronize(cudaStreamLegacy));  // see copies_done (engine.cu)
  return Status();
}

// A page-locked block of host memory that kernels can write, for the time of a
// transfer. Page-locking takes 1 to 5 ms whatever the size, so up to
// POOL_MOST blocks that are not in use are kept for the process's later
// transfers, of any batch, thread or device.
struct PinnedBlock {
  static constexpr size_t BYTES = 2 << 20, POOL_MOST = 4;
  void* p = nullptr;
  cudaError_t error = cudaSuccess;
  PinnedBlock() {
    {
      std::lock_guard<std::mutex> hold(pool().lock);
      if (!pool().free.empty()) {
        p = pool().free.back();
        pool().free.pop_back();
      }
    }
    if (!p) error = cudaHostAlloc(&p, BYTES, cudaHostAllocPortable | cudaHostAllocMapped);
    if (error != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
  }
  ~PinnedBlock() {
    if (!p) return;
    {
      std::lock_guard<std::mutex> hold(pool().lock);
      if (pool().free.size() < POOL_MOST) {
        pool().free.push_back(p);
        return;
      }
    }
    cudaFreeHost(p);
  }
  PinnedBlock(const PinnedBlock&) = delete;
  PinnedBlock& operator=(const PinnedBlock&) = delete;

 private:
  struct Pool {
    std::mutex lock;
    std::vector<void*> free;
    Pool() { free.reserve(POOL_MOST); }
  };
  // Never destroyed: a batch may be closed while the process exits.
  static Pool& pool() {
    static Pool* const the = new Pool();
    return *the;
  }
};
// A node has at most 16 actions of 1326 hands.
static_assert(sizeof(StorageBlockD) + 2 * 16 * DCFR_NUM_COMBOS * sizeof(float) <= PinnedBlock::BYTES, "a node fits");

// Slices (spot x 32 hands) up to which a block's warps share one; terminals
// per SM, and groups per block, up to which each terminal takes a block.
constexpr int BATCH_SHARE_ITEMS = 148 * 24;
constexpr int BATCH_BLOCK_TASKS_PER_SM = 4, BATCH_BLOCK_GROUPS = 5;

inline int pad8(int n) { return (n + 7) & ~7; }

}  // namespace

struct Batch::Impl {
  std::vector<Game> games;
  std::vector<SpotD> spots;
  std::vector<uint64_t> store;                  // per spot: float offset of its storage
  std::vector<std::vector<uint64_t>> node_off;  // per spot, per node: float offset of a player block in the spot
  std::vector<uint64_t> spot_len;               // storage floats per spot
  std::vector<double> cost;
  int maxa = 1, max_slots = 1, stride = 8, tstride = 1, cstride = 8, emax = 1;
  bool share = false;       // row passes: RowShape
  int row_blocks = 0;
  uint64_t total_store = 0, total_slots = 0;
  bool staged = true;  // row passes: plan records in shared memory
  size_t ntasks[2] = {0, 0}, nunits[2] = {0, 0}, ndown[2] = {0, 0};
  int max_up[2] = {0, 0}, max_down[2] = {0, 0};
  // Device.
  cudaStream_t stream = nullptr;
  float *regrets = nullptr, *sums = nullptr, *reach = nullptr, *vals = nullptr, *roots = nullptr, *root_out = nullptr;
  uint32_t* alive = nullptr;  // [2][total_slots]
  uint8_t *hc1 = nullptr, *hc2 = nullptr;
  uint32_t* same = nullptr;
  int4* dims = nullptr;
  uint16_t *cat = nullptr, *seg = nullptr;
  uint4* rec = nullptr;
  EntryD* tables = nullptr;
  uint32_t* tcount = nullptr;
  uint8_t* boards = nullptr;
  SegDown* down[2] = {nullptr, nullptr};
  SegUp* up[2] = {nullptr, nullptr};
  uint32_t* levs[2] = {nullptr, nullptr};
  uint8_t* deferred[2] = {nullptr, nullptr};
  FastTask* term[2] = {nullptr, nullptr};
  TermUnit* units[2] = {nullptr, nullptr};
  SpotD* d_spots = nullptr;
  RowItem *items_lpt = nullptr, *items_nat = nullptr;
  DiscountD* disc = nullptr;
  DiscountD* cur_disc = nullptr;
  uint32_t disc_len = 0;
  uint32_t* counter = nullptr;
  uint32_t iterations = 0;
  dcfr_batch_tuning tuning{};
  cudaGraphExec_t graph = nullptr;
  uint32_t graph_iters = 0;
  int sms = 148, optin = 0;
  int max_groups = 0, group_warps = 2, block_blocks = 0;  // group kernel: groups per block; block kernel: blocks
  uint64_t launches = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  double last_ms = 0.0;

  ~Impl();
  Status init(const dcfr_config* cfgs, int count);
  int occupancy(int warps) const;
  bool by_blocks(int p) const;
  void enqueue_rows(int mode, int up_p, int down_p, bool lpt, float* out, bool next = false);
  void enqueue_terminals(int p, const dcfr_batch_tuning& t, const PassTurn& turn = PassTurn());
  void enqueue_start(bool advance);
  Status launch_evaluation(int mode, const dcfr_batch_tuning& t);
  void enqueue_iteration(bool first, bool last);
  Status ensure_discounts(uint32_t max_t);
  Status capture(uint32_t iters);
  Status run(uint32_t n);
};

// Kernels of one iteration of every spot, and those before the first.
constexpr uint64_t BATCH_LAUNCHES = 4, BATCH_START = 2;

Batch::Impl::~Impl() {
  if (stream) cudaStreamSynchronize(stream);
  if (graph) cudaGraphExecDestroy(graph);
  bfree(regrets);
  bfree(sums);
  bfree(reach);
  bfree(vals);
  bfree(roots);
  bfree(root_out);
  bfree(hc1);
  bfree(hc2);
  bfree(same);
  bfree(cat);
  bfree(seg);
  bfree(rec);
  bfree(tables);
  bfree(tcount);
  bfree(boards);
  bfree(alive);
  bfree(dims);
  for (int p = 0; p < 2; p++) {
    bfree(down[p]);
    bfree(up[p]);
    bfree(levs[p]);
    bfree(deferred[p]);
    bfree(term[p]);
    bfree(units[p]);
  }
  bfree(cur_disc);
  bfree(d_spots);
  bfree(items_lpt);
  bfree(items_nat);
  bfree(disc);
  bfree(counter);
  if (ev0) cudaEventDestroy(ev0);
  if (ev1) cudaEventDestroy(ev1);
  if (stream) cudaStreamDestroy(stream);
}

// DcfrParams -> Discount (cfr.rs:86-106); defined in engine.cu.
DiscountD discount_of(uint32_t t, const dcfr_params& prm);

Status Batch::Impl::ensure_discounts(uint32_t max_t) {
  if (disc && max_t < disc_len) return Status();
  const uint32_t len = std::max<uint32_t>(max_t + 1, disc_len * 2);
  std::vector<DiscountD> tab(len);
  for (uint32_t t = 0; t < len; t++) tab[t] = discount_of(t, games[0].cfg.dcfr);
  BK(cudaStreamSynchronize(stream));
  if (graph) {
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  bfree(disc);
  Status s = upload(disc, tab, "discounts");
  disc_len = len;
  return s;
}

Status Batch::Impl::init(const dcfr_config* cfgs, int count) {
  Status s;
  BK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  BK(cudaEventCreate(&ev0));
  BK(cudaEventCreate(&ev1));
  int dev = 0;
  BK(cudaGetDevice(&dev));
  BK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  games.resize(count);
  for (int i = 0; i < count; i++) {
    const dcfr_config& c = cfgs[i];
    if (c.board_len != 5 || c.root.street != DCFR_RIVER) {
      s.code = DCFR_ERR_UNSUPPORTED;
      s.msg = "spot " + std::to_string(i) + ": the batched solve takes river spots (5-card board, river root)";
      return s;
    }
    if (c.precision != DCFR_PRECISION_FAST) {
      s.code = DCFR_ERR_UNSUPPORTED;
      s.msg = "spot " + std::to_string(i) + ": the batched solve runs in fast precision";
      return s;
    }
    if (std::memcmp(&c.dcfr, &cfgs[0].dcfr, sizeof c.dcfr) != 0) {
      s.code = DCFR_ERR_INVALID_ARG;
      s.msg = "spot " + std::to_string(i) + ": all spots of a batch share one DcfrParams";
      return s;
    }
    std::string msg;
    int rc = build_game(c, games[i], msg, true);
    if (rc) {
      s.code = rc;
      s.msg = "spot " + std::to_string(i) + ": " + msg;
      return s;
    }
    if (games[i].compressed) {
      s.code = DCFR_ERR_UNSUPPORTED;
      s.msg = "spot " + std::to_string(i) + ": the batched solve runs f32 storage";
      return s;
    }
  }
  // Host plans and the layout of every device array: slots, value rows and
  // terminal tasks numbered over all spots.
  std::vector<SegDown> hdown[2];
  std::vector<SegUp> hup[2];
  std::vector<uint32_t> hlevs[2];
  std::vector<FastTask> hterm[2];
  std::vector<TermUnit> hunits[2];
  std::vector<uint8_t> h1, h2, hb;
  std::vector<uint32_t> hs;
  std::vector<float> hroot;
  std::vector<int4> hdims;
  uint64_t vals_len = 0, reach_len = 0;  // entries
  int slices = 0;                         // of 32 hands
  spots.resize(count);
  store.resize(count);
  node_off.resize(count);
  spot_len.resize(count);
  cost.resize(count);
  for (int i = 0; i < count; i++) tstride = std::max(tstride, std::max(games[i].n[0], games[i].n[1]));
  cstride = (3 * tstride + 7) / 8 * 8;
  stride = std::max(8, pad8(tstride));
  emax = fast_emax(tstride);
  for (int i = 0; i < count; i++) {
    const Game& g = games[i];
    SpotD& S = spots[i];
    std::memset(&S, 0, sizeof S);
    const int hp0 = pad8(g.n[0]), hp1 = pad8(g.n[1]);
    S.hp[0] = hp0;
    S.hp[1] = hp1;
    hdims.push_back(make_int4(g.n[0], g.n[1], hp0, hp1));
    const size_t N = g.nodes.size();
    // Storage: player blocks [a][hp_q] in the reference's node order.
    const std::vector<uint32_t> players = players_in_storage_order(g);
    node_off[i].assign(N, 0);
    uint64_t len = 0;
    for (uint32_t v : players) {
      node_off[i][v] = len;
      len += (uint64_t)g.nodes[v].nchild * (uint64_t)(g.nodes[v].player ? hp1 : hp0);
      maxa = std::max<int>(maxa, g.nodes[v].nchild);
    }
    store[i] = total_store;
    spot_len[i] = len;
    total_store += len;
    // Hands, identical-hand maps, root rows, board.
    for (int q = 0; q < 2; q++)
      for (int h = 0; h < stride; h++) {
        const bool in = h < g.n[q];
        h1.push_back(in ? g.c1[q][h] : 255);
        h2.push_back(in ? g.c2[q][h] : 255);
        hs.push_back(in ? g.same[q][h] : NONE32);
      }
    for (int p = 0; p < 2; p++)
      for (int h = 0; h < stride; h++) hroot.push_back(h < g.n[p ^ 1] ? g.weights[p ^ 1][h] : 0.0f);
    for (int k = 0; k < 5; k++) hb.push_back((uint8_t)g.board[k]);
    S.stride = std::max(ROW_UNIT, std::max(hp0, hp1));
    S.slot = (uint32_t)total_slots;
    S.reach = (uint32_t)(reach_len / ROW_UNIT);
    S.vals = (uint32_t)(vals_len / ROW_UNIT);
    const uint32_t units = (uint32_t)(S.stride / ROW_UNIT);  // of a row
    slices += (S.stride + 31) / 32;
    const uint32_t layout = (uint32_t)(2 * i);
    // Traversal plans: slots, down tasks (breadth first), up tasks (deepest
    // first), terminals (showdowns with paired folds, and folds on the same
    // layout: see build_plan, engine.cu).
    uint64_t work_units = 0;
    for (int p = 0; p < 2; p++) {
      const int o = p ^ 1;
      const uint32_t entries = (uint32_t)S.hp[o];
      std::vector<uint32_t> slot(N, 0), depth(N, 0);
      std::vector<std::vector<SegUp>> ups;
      std::vector<std::vector<SegDown>> downs;
      std::vector<FastTask> sds, folds;
      uint32_t next_slot = 1;
      std::vector<uint32_t> queue{0};
      for (size_t qi = 0; qi < queue.size(); qi++) {
        const uint32_t v = queue[qi];
        const GNode& nd = g.nodes[v];
        const uint32_t sv = slot[v];
        if (nd.kind == N_PLAYER) {
          const bool own = nd.player == p;
          const uint32_t first_slot = own ? sv : next_slot;
          if (!own) next_slot += nd.nchild;
          for (uint32_t c = 0; c < nd.nchild; c++) {
            slot[nd.first + c] = own ? sv : first_slot + c;
            depth[nd.first + c] = depth[v] + 1;
            queue.push_back(nd.first + c);
          }
          if (ups.size() <= depth[v]) ups.resize(depth[v] + 1), downs.resize(depth[v] + 1);
          const uint64_t at = store[i] + node_off[i][v];
          const float uniform = 1.0f / (float)nd.nchild;
          if (!own) downs[depth[v]].push_back(SegDown{sv, first_slot, nd.nchild, 0, at, S.reach + first_slot * units, uniform});
          ups[depth[v]].push_back(SegUp{own ? (uint32_t)U_OWN : (uint32_t)U_OPP_SUM, nd.nchild, sv, S.vals + v * units,
                                        S.vals + nd.first * units, first_slot, 0, S.vals + v * units, at, uniform, 0});
          work_units += nd.nchild;
        } else if (nd.kind == N_FOLD || nd.kind == N_SHOWDOWN) {
          // Every terminal of a river spot sits below a river decision node:
          // batched evaluation (cfr.rs:282-284, river.rs:163-249), with a fold
          // beside a showdown under the traverser's own decision read off the
          // showdown's sums.
          const GNode& par = g.nodes[nd.parent];
          const double hpot = g.half_pot, norm = g.norm;
          if (nd.kind == N_FOLD) {
            bool paired = false;
            if (par.player == p)
              for (uint32_t c = par.first; c < par.first + par.nchild; c++)
                if (g.nodes[c].kind == N_SHOWDOWN) paired = true;
            if (paired) continue;
            const int f = nd.player;
            const double val = f == p ? -(hpot + (double)nd.invest[p]) : hpot + (double)nd.invest[f] - (double)nd.rake;
            folds.push_back(FastTask{T_FOLD_BATCH, layout, S.slot + sv, S.vals + v * units, NONE32, S.reach + sv * units,
                                     entries, 0, val * norm, 0.0, 0.0, 0.0});
          } else {
            const double rake = (double)nd.rake;
            FastTask t{T_SHOWDOWN_BATCH, layout, S.slot + sv, S.vals + v * units, NONE32, S.reach + sv * units, entries, 0,
                       (hpot + (double)nd.invest[o] - rake) * norm, -(hpot + (double)nd.invest[p]) * norm,
                       0.5 * ((double)(nd.invest[o] - nd.invest[p]) - rake) * norm, 0.0};
            if (par.player == p)
              for (uint32_t c = par.first; c < par.first + par.nchild; c++)
                if (g.nodes[c].kind == N_FOLD) {
                  const GNode& fn = g.nodes[c];
                  const int f = fn.player;
                  const double val =
                      f == p ? -(hpot + (double)fn.invest[p]) : hpot + (double)fn.invest[f] - (double)fn.rake;
                  t.frow = S.vals + c * units;
                  t.d = val * norm;
                }
            sds.push_back(t);
          }
        }
      }
      BatchPart& B = S.part[p];
      B.down_lev = (uint32_t)hlevs[p].size();
      B.ndown = (uint32_t)downs.size();
      for (const std::vector<SegDown>& l : downs) {
        hlevs[p].push_back((uint32_t)hdown[p].size());
        hdown[p].insert(hdown[p].end(), l.begin(), l.end());
      }
      hlevs[p].push_back((uint32_t)hdown[p].size());
      B.up_lev = (uint32_t)hlevs[p].size();
      B.nup = (uint32_t)ups.size();
      for (size_t l = ups.size(); l-- > 0;) {
        hlevs[p].push_back((uint32_t)hup[p].size());
        hup[p].insert(hup[p].end(), ups[l].begin(), ups[l].end());
      }
      hlevs[p].push_back((uint32_t)hup[p].size());
      // Showdowns and folds interleaved evenly (folds are cheaper, and blocks
      // take contiguous ranges).
      hunits[p].push_back(TermUnit{layout, (uint32_t)hterm[p].size(), (uint32_t)(sds.size() + folds.size()), 0});
      for (size_t x = 0, y = 0; x < sds.size() || y < folds.size();)
        if (y >= folds.size() || (x < sds.size() && x * folds.size() <= y * sds.size())) hterm[p].push_back(sds[x++]);
        else hterm[p].push_back(folds[y++]);
      S.nslots = std::max(S.nslots, next_slot);
      max_up[p] = std::max<int>(max_up[p], (int)(hup[p].size() - hlevs[p][B.up_lev]));
      max_down[p] = std::max<int>(max_down[p], (int)(hdown[p].size() - hlevs[p][B.down_lev]));
      work_units += sds.size() * 3 + folds.size();
    }
    max_slots = std::max<int>(max_slots, (int)S.nslots);
    total_slots += S.nslots;
    vals_len += N * S.stride;
    reach_len += (uint64_t)S.nslots * S.stride;
    cost[i] = (double)work_units * (double)S.stride;
  }
  if (max_slots > BATCH_MAX_SLOTS) {
    s.code = DCFR_ERR_UNSUPPORTED;
    s.msg = "a spot's tree needs more than " + std::to_string(BATCH_MAX_SLOTS) + " reach slots";
    return s;
  }
  if (std::max(vals_len, reach_len) / ROW_UNIT >= NONE32) {
    s.code = DCFR_ERR_UNSUPPORTED;
    s.msg = "the batch's rows pass what a 32-bit row number counts";
    return s;
  }
  // Device arrays.
  if (!(s = balloc(regrets, total_store, "batch storage")).ok()) return s;
  if (!(s = balloc(sums, total_store, "batch storage")).ok()) return s;
  BK(cudaMemsetAsync(regrets, 0, std::max<uint64_t>(total_store, 1) * 4, stream));
  BK(cudaMemsetAsync(sums, 0, std::max<uint64_t>(total_store, 1) * 4, stream));
  if (!(s = balloc(vals, vals_len, "batch value rows")).ok()) return s;
  if (!(s = balloc(reach, reach_len, "batch reach rows")).ok()) return s;
  if (!(s = balloc(alive, 2 * total_slots, "batch liveness flags")).ok()) return s;
  BK(cudaMemsetAsync(vals, 0, std::max<uint64_t>(vals_len, 1) * 4, stream));
  BK(cudaMemsetAsync(reach, 0, std::max<uint64_t>(reach_len, 1) * 4, stream));
  if (!(s = upload(hc1, h1, "batch hands")).ok()) return s;
  if (!(s = upload(hc2, h2, "batch hands")).ok()) return s;
  if (!(s = upload(same, hs, "batch hands")).ok()) return s;
  if (!(s = upload(dims, hdims, "batch hands")).ok()) return s;
  if (!(s = upload(roots, hroot, "batch root rows")).ok()) return s;
  if (!(s = balloc(root_out, hroot.size(), "batch root rows")).ok()) return s;
  if (!(s = upload(boards, hb, "batch boards")).ok()) return s;
  for (int p = 0; p < 2; p++) {
    ntasks[p] = hterm[p].size();
    nunits[p] = hunits[p].size();
    ndown[p] = hdown[p].size();
    if (!(s = upload(down[p], hdown[p], "batch plan")).ok()) return s;
    if (!(s = upload(up[p], hup[p], "batch plan")).ok()) return s;
    if (!(s = upload(levs[p], hlevs[p], "batch plan")).ok()) return s;
    if (!(s = upload(term[p], hterm[p], "batch plan")).ok()) return s;
    if (!(s = upload(units[p], hunits[p], "batch plan")).ok()) return s;
    if (!(s = balloc(deferred[p], hdown[p].size() * ((stride + 31) / 32), "batch plan")).ok()) return s;
  }
  if (!(s = upload(d_spots, spots, "batch plan")).ok()) return s;
  // The row passes' blocks, spots in input order and longest first. A block's
  // warps share a slice while there are too few slices to give every warp its
  // own (us an iteration, shared against not: 37 spots of 34 slices 152 against
  // 334, 512 spots 2113 against 1347).
  share = slices <= BATCH_SHARE_ITEMS;
  std::vector<uint32_t> order(count);
  std::iota(order.begin(), order.end(), 0u);
  auto items = [&] {
    const int hands = share ? RowShape<true>::SLICE : RowShape<false>::SLICE;
    const int per = share ? RowShape<true>::SLICES : RowShape<false>::SLICES;
    std::vector<RowItem> v;
    for (uint32_t i : order)
      for (int sl = 0; sl * hands < spots[i].stride; sl += per) v.push_back(RowItem{i, (uint32_t)sl});
    return v;
  };
  row_blocks = (int)items().size();
  if (!(s = upload(items_nat, items(), "batch order")).ok()) return s;
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return cost[a] > cost[b]; });
  if (!(s = upload(items_lpt, items(), "batch order")).ok()) return s;
  // Strength tables and scan layouts, per spot (its board and fold layouts).
  if (!(s = balloc(tables, (size_t)count * 2 * tstride, "batch strength tables")).ok()) return s;
  if (!(s = balloc(tcount, (size_t)count * 2, "batch strength tables")).ok()) return s;
  const size_t nl = (size_t)count * 2 * 2;
  if (!(s = balloc(cat, nl * cstride, "batch scan layouts")).ok()) return s;
  if (!(s = balloc(seg, nl * FAST_SEGS, "batch scan layouts")).ok()) return s;
  if (!(s = balloc(rec, nl * tstride, "batch scan layouts")).ok()) return s;
  for (int i = 0; i < count; i++) {
    const Game& g = games[i];
    const uint8_t* a0 = hc1 + (size_t)i * 2 * stride;
    const uint8_t* b0 = hc2 + (size_t)i * 2 * stride;
    const uint8_t* a1 = a0 + stride;
    const uint8_t* b1 = b0 + stride;
    EntryD* tb = tables + (size_t)i * 2 * tstride;
    uint32_t* tc = tcount + (size_t)i * 2;
    launch_strength(boards + (size_t)i * 5, 1, a0, b0, a1, b1, g.n[0], g.n[1], tb, tc, tstride, stream);
    launch_fast_layouts(tb, tc, tstride, 1, a0, b0, a1, b1, g.n[0], g.n[1], cat + (size_t)i * 4 * cstride,
                        seg + (size_t)i * 4 * FAST_SEGS, rec + (size_t)i * 4 * tstride, cstride, stream);
  }
  BK(cudaGetLastError());
  if (!(s = balloc(counter, 1, "batch counter")).ok()) return s;
  if (!(s = balloc(cur_disc, 2, "batch counter")).ok()) return s;
  BK(cudaMemsetAsync(counter, 0, 4, stream));
  if (!(s = ensure_discounts(1024)).ok()) return s;
  BK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  staged = RowSmem(std::max(max_up[0], max_up[1]), std::max(max_down[0], max_down[1]), std::max(max_down[0], max_down[1]),
                   max_slots, RowShape<false>::SLICES)
               .total <= (size_t)optin;
  for (int mode : {M_CFR, M_BR, M_AVG})
    for (const void* fn : {row_fn<true>(mode, maxa, staged), row_fn<false>(mode, maxa, staged)})
      BK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
  int bps = 0;
  max_groups = group_terminal_setup(stride, cstride, tstride, group_warps, bps, true);
  const int fast_bps = fast_blocks_per_sm(stride, emax, cstride, tstride, true);
  if (max_groups <= 0 || fast_bps <= 0) {
    s.code = DCFR_ERR_UNSUPPORTED;
    s.msg = "batched kernel: a spot's layout does not fit in shared memory";
    return s;
  }
  block_blocks = sms * fast_bps;
  // Default tuning until autotune: the most terminals in flight.
  for (int w = 1; w <= BATCH_MAX_THREADS / 32; w++)
    if (tuning_smem(stride, cstride, tstride, max_slots, w) <= (size_t)optin) tuning.warps = w;
  tuning.blocks_per_sm = occupancy(tuning.warps);
  tuning.iterations_per_launch = 25;
  tuning.longest_first = 1;
  BK(cudaStreamSynchronize(stream));
  return Status();
}

// Resident blocks per SM of the group terminal kernel with up to `warps`
// terminals in flight in a block.
int Batch::Impl::occupancy(int warps) const {
  return std::max(1, group_terminal_occupancy(stride, cstride, tstride, std::min(warps, max_groups), group_warps, true));
}

// A row pass over all spots: the up pass of traverser up_p, then the down
// pass of down_p (-1: not wanted).
void Batch::Impl::enqueue_rows(int mode, int up_p, int down_p, bool lpt, float* out, bool next) {
  BatchPass P{};
  P.spots = d_spots;
  P.items = lpt ? items_lpt : items_nat;
  P.stride = stride;
  P.max_slots = max_slots;
  P.regrets = regrets;
  P.sums = sums;
  P.reach = reach;
  P.vals = vals;
  P.alive[0] = alive;
  P.alive[1] = alive + total_slots;
  P.disc = cur_disc;
  P.down_disc = cur_disc + (next ? 1 : 0);
  P.up_p = up_p;
  P.down_p = down_p;
  if (up_p >= 0) {
    P.up = up[up_p];
    P.fix = down[up_p];
    P.up_levs = levs[up_p];
    P.up_deferred = deferred[up_p];
    P.max_up = staged ? max_up[up_p] : 0;
    P.max_fix = staged && mode == M_CFR ? max_down[up_p] : 0;
    P.n_fix = (uint32_t)ndown[up_p];
    P.root_out = out;
  }
  if (down_p >= 0) {
    P.down = down[down_p];
    P.down_levs = levs[down_p];
    P.down_deferred = deferred[down_p];
    P.roots = roots;
    P.max_down = staged ? max_down[down_p] : 0;
    P.n_down = (uint32_t)ndown[down_p];
  }
  const int per = share ? RowShape<true>::SLICES : RowShape<false>::SLICES;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)row_blocks);
  cfg.blockDim = dim3((unsigned)((share ? RowShape<true>::WARPS : RowShape<false>::WARPS) * 32));
  cfg.dynamicSmemBytes = RowSmem(P.max_up, P.max_fix, P.max_down, P.max_slots, per).total;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void* params[] = {(void*)&P};
  cudaLaunchKernelExC(&cfg, share ? row_fn<true>(mode, maxa, staged) : row_fn<false>(mode, maxa, staged),
                      params);
}

// Whether a traversal's terminals take a block each: while there are few of
// them or hand lists so long that few groups fit a block (1081 hands, five
// groups, us an iteration, block against group kernel: 37 spots 126 against 135,
// 512 spots 1148 against 1134). Otherwise two warps each.
bool Batch::Impl::by_blocks(int p) const {
  return max_groups <= BATCH_BLOCK_GROUPS || ntasks[p] <= (size_t)BATCH_BLOCK_TASKS_PER_SM * sms;
}

// All spots' terminals of one traversal.
void Batch::Impl::enqueue_terminals(int p, const dcfr_batch_tuning& t, const PassTurn& turn) {
  FastArgs F;
  F.turn = turn;
  F.reach = reach;
  F.vals = vals;
  F.alive = alive + (size_t)p * total_slots;
  F.cat = cat;
  F.seg = seg;
  F.rec = rec;
  F.same = same;
  F.dims = dims;
  F.cstride = cstride;
  F.tstride = tstride;
  F.emax = emax;
  F.n[0] = F.n[1] = tstride;
  F.hp[0] = F.hp[1] = stride;
  F.stride = stride;
  F.p = p;
  if (by_blocks(p)) {
    launch_fast_terminal(F, term[p], (int)ntasks[p], block_blocks, stream);
    return;
  }
  launch_group_terminal(F, term[p], units[p], (int)nunits[p], (int)ntasks[p], std::min(t.warps, max_groups), group_warps,
                        sms * std::max(t.blocks_per_sm, 1), stream);
}

// Before a run's first down pass: flags cleared, and the iteration stepped.
void Batch::Impl::enqueue_start(bool advance) {
  launch_traversal_start(alive, (int)total_slots, alive + total_slots, (int)total_slots, reach, roots, 0,
                         advance ? counter : nullptr, disc, disc_len, cur_disc, nullptr, stream);
}

// One best-response or average pair of traversals of every spot.
Status Batch::Impl::launch_evaluation(int mode, const dcfr_batch_tuning& t) {
  const bool lpt = t.longest_first != 0;
  enqueue_start(false);
  enqueue_rows(mode, -1, 0, lpt, nullptr);
  enqueue_terminals(0, t);
  enqueue_rows(mode, 0, 1, lpt, root_out);
  enqueue_terminals(1, t);
  enqueue_rows(mode, 1, -1, lpt, root_out);
  BK(cudaGetLastError());
  launches += BATCH_START + 4;
  return Status();
}

// An iteration after its first traversal's down pass. The up pass of the
// second traversal is one launch with the next iteration's first down pass,
// and the terminal kernels do what a start kernel would (PassTurn), as in
// Engine::enqueue_rolled (us an iteration against separate ones: 37 spots 113
// to 105, 512 spots 1018 to 1011 then).
void Batch::Impl::enqueue_iteration(bool first, bool last) {
  const bool lpt = tuning.longest_first != 0;
  PassTurn turn;
  turn.counter = counter;
  turn.table = disc;
  turn.table_len = disc_len;
  turn.cur = cur_disc;
  turn.clear = alive + total_slots;
  turn.nclear = first ? 0 : (uint32_t)total_slots;
  turn.step = first ? TURN_KEEP : TURN_BEGIN;
  enqueue_terminals(0, tuning, turn);
  enqueue_rows(M_CFR, 0, 1, lpt, nullptr);
  turn.clear = alive;
  turn.nclear = last ? 0 : (uint32_t)total_slots;
  turn.step = last ? TURN_KEEP : TURN_NEXT;
  enqueue_terminals(1, tuning, turn);
  enqueue_rows(M_CFR, 1, last ? -1 : 0, lpt, nullptr, !last);
}

Status Batch::Impl::capture(uint32_t iters) {
  if (graph && graph_iters == iters) return Status();
  if (graph) {
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  cudaGraph_t g;
  BK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
  for (uint32_t i = 0; i < iters; i++) enqueue_iteration(false, false);
  BK(cudaStreamEndCapture(stream, &g));
  const cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
  cudaGraphDestroy(g);
  BK(e);
  graph_iters = iters;
  BK(cudaGraphUpload(graph, stream));
  return Status();
}

// n iterations: all but the first and the last, and fewer than a graph's left
// over, in graphs.
Status Batch::Impl::run(uint32_t n) {
  Status s;
  if (!(s = ensure_discounts(iterations + n + 1)).ok()) return s;
  const uint32_t k = std::max<uint32_t>(tuning.iterations_per_launch, 1);
  if (n >= 2 && n - 2 >= k && !(s = capture(k)).ok()) return s;
  BK(cudaEventRecord(ev0, stream));
  if (n > 0) {
    enqueue_start(true);
    enqueue_rows(M_CFR, -1, 0, tuning.longest_first != 0, nullptr);
    launches += BATCH_START + (uint64_t)n * BATCH_LAUNCHES;
  }
  for (uint32_t i = 0; i < n;) {
    if (i > 0 && n - 1 - i >= k) {
      BK(cudaGraphLaunch(graph, stream));
      i += k;
    } else {
      enqueue_iteration(i == 0, i + 1 == n);
      i++;
    }
  }
  BK(cudaGetLastError());
  BK(cudaEventRecord(ev1, stream));
  BK(cudaEventSynchronize(ev1));
  float ms = 0.0f;
  BK(cudaEventElapsedTime(&ms, ev0, ev1));
  last_ms = ms;
  iterations += n;
  return Status();
}

Batch::Batch() : impl_(new Impl()) {}
Batch::~Batch() = default;

Status Batch::create(const dcfr_config* cfgs, int count, std::unique_ptr<Batch>& out) {
  Status s;
  if (count <= 0) {
    s.code = DCFR_ERR_INVALID_ARG;
    s.msg = "a batch has at least one spot";
    return s;
  }
  std::unique_ptr<Batch> b(new Batch());
  if (!(s = b->impl_->init(cfgs, count)).ok()) return s;
  out = std::move(b);
  return Status();
}

int Batch::count() const { return (int)impl_->spots.size(); }
uint32_t Batch::iterations() const { return impl_->iterations; }
double Batch::last_iterate_ms() const { return impl_->last_ms; }
uint64_t Batch::kernel_launches() const { return impl_->launches; }
dcfr_batch_tuning Batch::tuning() const { return impl_->tuning; }

double Batch::iteration_bytes() const {
  double b = 0.0;
  for (const Game& g : impl_->games)
    b += 20.0 * (double)g.storage_len + 2.0 * (double)g.nodes.size() * 4.0 * ((double)g.n[0] + (double)g.n[1]);
  return b;
}

Status Batch::iterate(uint32_t n) { return impl_->run(n); }

Status Batch::set_tuning(const dcfr_batch_tuning& t) {
  Impl& I = *impl_;
  Status s;
  if (t.warps < 1 || t.warps > BATCH_MAX_THREADS / 32 ||
      tuning_smem(I.stride, I.cstride, I.tstride, I.max_slots, t.warps) > (size_t)I.optin ||
      t.iterations_per_launch < 1) {
    s.code = DCFR_ERR_INVALID_ARG;
    s.msg = "batch tuning: warps, shared memory or iterations per launch out of range";
    return s;
  }
  const int b = I.occupancy(t.warps);
  dcfr_batch_tuning u = t;
  u.blocks_per_sm = std::max(1, std::min(t.blocks_per_sm > 0 ? t.blocks_per_sm : b, b));
  I.tuning = u;
  if (I.graph) {
    cudaGraphExecDestroy(I.graph);
    I.graph = nullptr;
  }
  return Status();
}

// The project's autotuner: times each candidate (warps per block, blocks per
// SM, iterations per launch, longest-first or natural order) from a snapshot of
// the storage, restores the snapshot and the iteration counter after every trial,
// and keeps the fastest candidate and its graph. A trial is two iterations more
// than trial_iterations: the first and the last of a run are never in a graph.
// Warps and blocks are a dimension only where a group kernel runs the terminals.
Status Batch::autotune(uint32_t trial_iterations, dcfr_batch_tuning& best) {
  Impl& I = *impl_;
  Status s;
  const uint64_t n = std::max<uint64_t>(I.total_store, 1);
  struct Held {
    float *regrets = nullptr, *sums = nullptr;
    cudaGraphExec_t graph = nullptr;
    ~Held() {
      bfree(regrets);
      bfree(sums);
      if (graph) cudaGraphExecDestroy(graph);
    }
  } held;
  if (!(s = balloc(held.regrets, n, "autotune snapshot")).ok()) return s;
  if (!(s = balloc(held.sums, n, "autotune snapshot")).ok()) return s;
  BK(cudaMemcpyAsync(held.regrets, I.regrets, n * 4, cudaMemcpyDeviceToDevice, I.stream));
  BK(cudaMemcpyAsync(held.sums, I.sums, n * 4, cudaMemcpyDeviceToDevice, I.stream));
  const uint32_t t_saved = I.iterations;
  const dcfr_batch_tuning saved = I.tuning;
  std::vector<dcfr_batch_tuning> cands;
  const uint32_t trial = std::max<uint32_t>(trial_iterations, 1), run = trial + 2;
  if (!(s = I.ensure_discounts(t_saved + run + 1)).ok()) return s;
  const bool groups = !I.by_blocks(0) || !I.by_blocks(1);
  for (int w = groups ? 2 : saved.warps; w <= BATCH_MAX_THREADS / 32; w++) {
    if (tuning_smem(I.stride, I.cstride, I.tstride, I.max_slots, w) > (size_t)I.optin) break;
    if (groups && w > 2 && w > I.max_groups) break;  // no more terminals in flight than at the last candidate
    for (uint32_t ipl : {trial, std::max<uint32_t>(trial / 5, 1u)})
      for (int lpt : {1, 0}) {
        dcfr_batch_tuning t{};
        t.warps = w;
        t.blocks_per_sm = I.occupancy(w);
        t.iterations_per_launch = ipl;
        t.longest_first = lpt;
        cands.push_back(t);
      }
    if (!groups) break;
  }
  double best_ms = 1e300;
  best = saved;
  for (const dcfr_batch_tuning& t : cands) {
    if (!(s = set_tuning(t)).ok()) break;
    if (!(s = I.run(run)).ok()) break;
    const double ms = I.last_ms * (double)trial / (double)run;
    if (ms < best_ms) {
      best_ms = ms;
      best = I.tuning;
      std::swap(held.graph, I.graph);
    }
    BK(cudaMemcpyAsync(I.regrets, held.regrets, n * 4, cudaMemcpyDeviceToDevice, I.stream));
    BK(cudaMemcpyAsync(I.sums, held.sums, n * 4, cudaMemcpyDeviceToDevice, I.stream));
    BK(cudaMemcpyAsync(I.counter, &t_saved, 4, cudaMemcpyHostToDevice, I.stream));
    BK(cudaStreamSynchronize(I.stream));
    I.iterations = t_saved;
  }
  if (!s.ok()) {
    set_tuning(saved);
    return s;
  }
  best.trial_ms = best_ms;
  best.candidates = (int)cands.size();
  if (!(s = set_tuning(best)).ok()) return s;
  std::swap(held.graph, I.graph);
  I.graph_iters = best.iterations_per_launch;
  return Status();
}

Status Batch::root_values(int mode, std::vector<double>& out) {
  Impl& I = *impl_;
  Status s;
  if (!(s = I.launch_evaluation(mode, I.tuning)).ok()) return s;
  std::vector<float> rows(I.spots.size() * 2 * I.stride);
  BK(cudaMemcpyAsync(rows.data(), I.root_out, rows.size() * 4, cudaMemcpyDeviceToHost, I.stream));
  BK(cudaStreamSynchronize(I.stream));
  out.assign(I.spots.size() * 2, 0.0);
  for (size_t i = 0; i < I.spots.size(); i++) {
    const Game& g = I.games[i];
    for (int p = 0; p < 2; p++) {
      double acc = -0.0;
      for (int h = 0; h < g.n[p]; h++) acc += (double)rows[(i * 2 + p) * I.stride + h] * (double)g.weights[p][h];
      out[2 * i + p] = acc;
    }
  }
  return Status();
}

Status Batch::exploitability(double* out) {
  std::vector<double> br, ev;
  Status s = root_values(M_BR, br);
  if (!s.ok()) return s;
  bool raked = false;
  for (const Game& g : impl_->games) raked |= g.cfg.rake_rate > 0.0 && g.cfg.rake_cap > 0.0;
  if (raked && !(s = root_values(M_AVG, ev)).ok()) return s;
  for (size_t i = 0; i < impl_->games.size(); i++) {
    const dcfr_config& c = impl_->games[i].cfg;
    if (c.rake_rate > 0.0 && c.rake_cap > 0.0)
      out[i] = ((br[2 * i] - ev[2 * i]) + (br[2 * i + 1] - ev[2 * i + 1])) / 2.0;
    else
      out[i] = (br[2 * i] + br[2 * i + 1]) / 2.0;
  }
  return Status();
}

Status Batch::storage_len(int spot, uint64_t& len) const {
  if (spot < 0 || spot >= count()) return Status{DCFR_ERR_INVALID_ARG, "spot index out of range"};
  len = impl_->games[spot].storage_len;
  return Status();
}

// One spot's storage, in the reference's layout: its decision nodes' records go
// into a page-locked block, the pack kernel reads them there and writes the
// nodes' cells beside them, and the host copies those to the caller's arrays;
// a large spot takes several rounds of whole nodes. Nothing of this belongs to
// the batch, so several threads may read spots of one batch, and the first
// read costs what a later one does. ms, a batch's first and later reads of a
// spot of 86,000 cells: with a table of all spots and buffers of the batch's own,
// made on the first read, 2.2 to 3.9 (512 spots: 3.8 to 86) and 0.11; now 0.12
// and 0.11.
Status Batch::download(int spot, float* regrets, float* sums) {
  Impl& I = *impl_;
  if (spot < 0 || spot >= count()) return Status{DCFR_ERR_INVALID_ARG, "spot index out of range"};
  const Game& g = I.games[spot];
  const std::vector<uint32_t> players = players_in_storage_order(g);
  const PinnedBlock lease;
  BK(lease.error);
  for (size_t i = 0; i < players.size();) {
    // The nodes that fit: a record and both kinds of cells of each.
    StorageBlockD* rec = static_cast<StorageBlockD*>(lease.p);
    const uint64_t from = g.nodes[players[i]].ref_offset;
    uint64_t len = 0;
    int nb = 0;
    for (; i < players.size(); i++, nb++) {
      const GNode& nd = g.nodes[players[i]];
      const uint64_t cells = (uint64_t)nd.nchild * (uint64_t)g.n[nd.player];
      if (nb > 0 && (nb + 1) * sizeof(StorageBlockD) + 2 * (len + cells) * sizeof(float) > PinnedBlock::BYTES) break;
      rec[nb] = StorageBlockD{I.store[spot] + I.node_off[spot][players[i]], nd.ref_offset - from, nd.nchild,
                              (uint32_t)g.n[nd.player], (uint32_t)I.spots[spot].hp[nd.player], 0};
      len += cells;
    }
    float* out[2] = {reinterpret_cast<float*>(rec + nb), reinterpret_cast<float*>(rec + nb) + len};
    if (regrets) launch_storage_pack(4, I.regrets, out[0], rec, nb, I.stream);
    if (sums) launch_storage_pack(4, I.sums, out[1], rec, nb, I.stream);
    BK(cudaGetLastError());
    BK(cudaStreamSynchronize(I.stream));
    if (regrets) std::memcpy(regrets + from, out[0], len * sizeof(float));
    if (sums) std::memcpy(sums + from, out[1], len * sizeof(float));
  }
  return Status();
}

}  // namespace dcfr
