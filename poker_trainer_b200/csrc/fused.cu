// Fused segments: one block walks the decision nodes of a street's subtree
// (FusedTree), every thread with the same 4 hands throughout, so a node's rows
// are produced and consumed by the same thread. The operations are those of
// down_item / up_item (row_items.cuh), in their order.
//
// With f32 storage and wide ranges the passes are bound by memory (a flop of
// 2456M cells, 468 hands: 6.3 TB/s of rows and storage); with 16-bit storage
// or short hand lists by how many nodes an SM has in flight, each a chain of
// task, liveness and storage reads. So a segment's tasks and liveness are kept
// in shared memory, and storage is copied there asynchronously: its 2 x 4
// rows of 4 cells a thread would take registers (80, six blocks of 128
// threads an SM; now at most 56, nine), and up passes copy the next node's
// rows while they work on one. us an iteration against loads into registers:
// flop of 873M cells, 16 bits, 468 hands 15365 to 12014; 2456M cells, f32,
// 34133 to 31082; 84M cells, sampled deals 1872 to 1762; turns of 14M and 6M
// cells 300 to 300 and 197 to 184.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "pdl.cuh"
#include "plan.hpp"
#include "row_items.cuh"

namespace dcfr {
namespace {

constexpr int LOCAL_SLOTS = 1 + FUSED_MAX_NODES * MAX_ACTIONS;

// An asynchronous copy of a thread's 4 cells (16 bytes of f32, 8 of 16-bit
// storage) into its own place of the stage; only that thread reads it.
template <int BYTES>
__device__ __forceinline__ void copy_async(void* smem, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A segment's tasks into shared memory (they are plan data).
template <typename Task>
__device__ __forceinline__ void load_tasks(Task* dst, const Task* src, uint32_t n) {
  static_assert(sizeof(Task) % 16 == 0, "16-byte loads");
  for (uint32_t i = threadIdx.x; i < n * (sizeof(Task) / 16); i += blockDim.x)
    reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
}

// Down: the opponent's nodes in BFS order, a barrier at every new level (it
// publishes the children's liveness, kept in shared memory by the slots'
// numbers in the segment, task.kind >> LOCAL_SHIFT).
template <int MODE, int MAXA, bool COMP>
__global__ void __launch_bounds__(ROW_MAX_THREADS, MAXA <= 4 ? 3 : 1) fused_down_kernel(RowArgs A, const FusedTree* __restrict__ trees,
                                                                     const DownTask* __restrict__ tasks, int maxa) {
  constexpr int E = COMP ? 8 : 16;  // bytes of 4 cells
  extern __shared__ uint4 stage_raw[];
  alignas(16) __shared__ DownTask st[FUSED_MAX_NODES];
  __shared__ uint8_t live[LOCAL_SLOTS];
  const FusedTree F = trees[blockIdx.x];
  load_tasks(st, tasks + F.down_first, F.down_count);
  for (int i = threadIdx.x; i < LOCAL_SLOTS; i += blockDim.x) live[i] = 0;
  const int tid = (int)threadIdx.x, lane = tid & 31, h0 = tid * VEC;
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  if (F.down_count == 0 || A.alive[st[0].in_slot] == 0) return;  // the segment's first opponent node holds its root's row
  const int o = A.p ^ 1, hp = pick(o, A.hp);
  const size_t stride = (size_t)A.stride;
  const bool valid = h0 < hp;
  const DiscountD d = MODE == M_CFR ? *A.disc : DiscountD{};
  // The thread's place for action a of the regrets (CFR) or sums; the sums
  // beside the regrets follow at `second`.
  const int step = (int)blockDim.x * E, second = maxa * step;
  char* mine = reinterpret_cast<char*>(stage_raw) + tid * E;
  int phase = 0;
  uint32_t out = 1;  // the task's first child, numbered in the segment
#pragma unroll 1
  for (uint32_t i = 0; i < F.down_count; i++) {
    const uint32_t kind = st[i].kind, in = kind >> LOCAL_SHIFT;
    const int na = (int)st[i].nchild;
    if (kind & LEVEL_BREAK) __syncthreads();
    const uint32_t lo = out;
    out += (uint32_t)na;
    if (in != 0 && live[in] == 0) continue;  // dead subtree: children stay dead
    const uint64_t store = st[i].store + h0;
    const uint32_t out_slot = st[i].out_slot, scale = st[i].cards;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 x[MAXA];
    float sdec = 0.0f;
    if (valid) {
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na) {
          const size_t e = store + (size_t)(a * hp);
          if constexpr (COMP) {
            copy_async<E>(mine + a * step, MODE == M_CFR ? (const void*)(A.rq + e) : (const void*)(A.sq + e));
            if (MODE == M_CFR) copy_async<E>(mine + second + a * step, A.sq + e);
          } else {
            copy_async<E>(mine + a * step, (MODE == M_CFR ? A.regrets : A.sums) + e);
            if (MODE == M_CFR) copy_async<E>(mine + second + a * step, A.sums + e);
          }
        }
      copy_commit();
      r = ld4(A.reach + (size_t)st[i].in_slot * stride + h0);
    }
    if constexpr (COMP) sdec = A.sscale[scale] / 65535.0f;
    copy_wait<0>();
    if (valid) {
      const float uniform = 1.0f / (float)na;
      float4 s, inv;
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na) {
          const char* q = mine + a * step;
          if constexpr (!COMP) x[a] = *reinterpret_cast<const float4*>(q);
          else if (MODE == M_CFR) x[a] = ldq(reinterpret_cast<const int16_t*>(q));
          else x[a] = scale4(ldq(reinterpret_cast<const uint16_t*>(q)), sdec);
#pragma unroll
          for (int j = 0; j < VEC; j++) {
            if (MODE == M_CFR) at(x[a], j) = max0(at(x[a], j));
            at(s, j) = a == 0 ? at(x[a], j) : at(s, j) + at(x[a], j);
          }
        }
#pragma unroll
      for (int j = 0; j < VEC; j++) at(inv, j) = recipf(at(s, j));
      // The strategy (regret_match_into, cfr.rs:161-192, or
      // normalize_in_place, cfr.rs:124-154).
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na)
#pragma unroll
          for (int j = 0; j < VEC; j++) at(x[a], j) = at(inv, j) == 0.0f ? uniform : at(x[a], j) * at(inv, j);
    }
    // Strategy sums s*gamma + sigma (or + sigma*reach) (cfr.rs:395-407); c is
    // the child's reach, sigma*reach.
    auto new_sum = [&](int a, float4 c) {
      float4 q;
      if constexpr (!COMP) q = *reinterpret_cast<const float4*>(mine + second + a * step);
      else q = scale4(ldq(reinterpret_cast<const uint16_t*>(mine + second + a * step)), sdec);
#pragma unroll
      for (int j = 0; j < VEC; j++) at(q, j) = at(q, j) * d.strat + (d.reach_weighted ? at(c, j) : at(x[a], j));
      return q;
    };
    auto child = [&](int a) {
      float4 c;
#pragma unroll
      for (int j = 0; j < VEC; j++) at(c, j) = at(x[a], j) * at(r, j);
      return c;
    };
    float smax = 0.0f;
    uint32_t any = 0;  // actions that some hand of the thread reaches
    if (valid) {
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na) {
          const float4 c = child(a);
          if constexpr (MODE == M_CFR) {
            const float4 q = new_sum(a, c);
            if constexpr (COMP) smax = fmaxf(smax, absmax4(q));
            else st4(A.sums + store + (size_t)(a * hp), q);
          }
          st4(A.reach + (size_t)(out_slot + a) * stride + h0, c);
          any |= nz4(c) ? 1u << a : 0u;
        }
    }
    any = __reduce_or_sync(0xffffffffu, any);
    if ((any >> lane) & 1u) {
      live[lo + lane] = 1;
      A.alive[out_slot + lane] = 1u;
    }
    if constexpr (COMP && MODE == M_CFR) {
      // The node's new scale and the re-encoded sums (storage.rs:315-328),
      // computed again from the stage.
      const float mx = block_max(smax, phase);
      const float sinv = mx > 0.0f ? 65535.0f / mx : 0.0f;
      if (valid) {
#pragma unroll
        for (int a = 0; a < MAXA; a++)
          if (a < na) {
            ushort4 q = make_ushort4(0, 0, 0, 0);
            if (mx > 0.0f) {
              const float4 s = new_sum(a, child(a));
              q = make_ushort4(enc_sum(s.x, sinv), enc_sum(s.y, sinv), enc_sum(s.z, sinv), enc_sum(s.w, sinv));
            }
            *reinterpret_cast<ushort4*>(A.sq + store + (size_t)(a * hp)) = q;
          }
      }
      if (tid == 0) A.sscale[scale] = mx;
    }
  }
}

// Up: all decision nodes, deepest level first. The storage of the next node is
// copied while a node is worked on (liveness is final, so it is known which
// nodes to skip).
template <int MODE, int MAXA, bool COMP>
__global__ void __launch_bounds__(ROW_MAX_THREADS, MAXA <= 4 ? 3 : 1) fused_up_kernel(RowArgs A, const FusedTree* __restrict__ trees,
                                                                   const UpTask* __restrict__ tasks, int maxa) {
  constexpr int E = COMP ? 8 : 16;
  extern __shared__ uint4 stage_raw[];
  alignas(16) __shared__ UpTask st[FUSED_MAX_NODES];
  __shared__ uint8_t live[FUSED_MAX_NODES];
  const FusedTree F = trees[blockIdx.x];
  load_tasks(st, tasks + F.up_first, F.up_count);
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  for (uint32_t i = threadIdx.x; i < F.up_count; i += blockDim.x) live[i] = A.alive[st[i].slot] != 0;
  __syncthreads();
  const int tid = (int)threadIdx.x, h0 = tid * VEC;
  const int p = A.p, hp = pick(p, A.hp);
  const size_t stride = (size_t)A.stride;
  const bool valid = h0 < hp;
  const DiscountD d = MODE == M_CFR ? *A.disc : DiscountD{};
  const int step = (int)blockDim.x * E;
  auto place = [&](uint32_t i, int a) {
    return reinterpret_cast<char*>(stage_raw) + (tid * E + ((i & 1) ? maxa * step : 0) + a * step);
  };
  auto fetch = [&](uint32_t i) {
    if (MODE != M_BR && i < F.up_count && valid && live[i] && (st[i].kind & KIND_MASK) == U_OWN) {
      const size_t e = st[i].store + h0;
      const int na = (int)st[i].nchild;
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na) {
          if constexpr (COMP)
            copy_async<E>(place(i, a), MODE == M_CFR ? (const void*)(A.rq + e + (size_t)(a * hp))
                                                     : (const void*)(A.sq + e + (size_t)(a * hp)));
          else
            copy_async<E>(place(i, a), (MODE == M_CFR ? A.regrets : A.sums) + e + (size_t)(a * hp));
        }
    }
    copy_commit();
  };
  int phase = 0;
  fetch(0);
#pragma unroll 1
  for (uint32_t i = 0; i < F.up_count; i++) {
    fetch(i + 1);
    if (!live[i]) continue;
    const int na = (int)st[i].nchild;
    const size_t child = (size_t)st[i].child;
    const bool own = (st[i].kind & KIND_MASK) == U_OWN;
    float4 v[MAXA];
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) {
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na) v[a] = ld4(A.vals + (child + a) * stride + h0);
    }
    if (!own) {
      // The sum of the live children, in child order.
      const uint32_t cs = st[i].child_slot;
      bool clive[MAXA];
#pragma unroll
      for (int a = 0; a < MAXA; a++) clive[a] = a < na && A.alive[cs + a] != 0;
      if (!valid) continue;
#pragma unroll
      for (int a = 0; a < MAXA; a++)
        if (a < na && clive[a])
#pragma unroll
          for (int j = 0; j < VEC; j++) at(out, j) += at(v[a], j);
    } else if constexpr (MODE == M_BR) {
      if (!valid) continue;
      out = v[0];
#pragma unroll
      for (int a = 1; a < MAXA; a++)
        if (a < na)
#pragma unroll
          for (int j = 0; j < VEC; j++) at(out, j) = at(v[a], j) > at(out, j) ? at(v[a], j) : at(out, j);
    } else {
      const float dec = !COMP ? 0.0f
                              : MODE == M_CFR ? A.rscale[st[i].cards] / 32767.0f : A.sscale[st[i].cards] / 65535.0f;
      copy_wait<1>();
      auto cell = [&](int a) {
        if constexpr (!COMP) return *reinterpret_cast<const float4*>(place(i, a));
        else if (MODE == M_CFR) return scale4(ldq(reinterpret_cast<const int16_t*>(place(i, a))), dec);
        else return scale4(ldq(reinterpret_cast<const uint16_t*>(place(i, a))), dec);
      };
      if constexpr (MODE == M_AVG) {
        if (!valid) continue;
        float4 s = cell(0), inv;
        for (int a = 1; a < na; a++) {
          float4 x = cell(a);
#pragma unroll
          for (int j = 0; j < VEC; j++) at(s, j) += at(x, j);
        }
        const float uniform = 1.0f / (float)na;
#pragma unroll
        for (int j = 0; j < VEC; j++) at(inv, j) = recipf(at(s, j));
#pragma unroll
        for (int a = 0; a < MAXA; a++)
          if (a < na) {
            float4 x = cell(a);
#pragma unroll
            for (int j = 0; j < VEC; j++) {
              const float sv = at(inv, j) == 0.0f ? uniform : at(x, j) * at(inv, j);
              at(out, j) += sv * at(v[a], j);
            }
          }
      } else {
        // own_node_update (cfr.rs:315-382).
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) {
#pragma unroll
          for (int a = 0; a < MAXA; a++)
            if (a < na) {
              float4 x = cell(a);
#pragma unroll
              for (int j = 0; j < VEC; j++) {
                const float y = max0(at(x, j));
                at(s, j) = a == 0 ? y : at(s, j) + y;
                at(out, j) += y * at(v[a], j);
              }
            }
#pragma unroll
          for (int j = 0; j < VEC; j++) {
            const float iv = recipf(at(s, j));
            at(out, j) *= iv;
            if (iv == 0.0f) {
              float m = -0.0f;
#pragma unroll
              for (int a = 0; a < MAXA; a++)
                if (a < na) m += at(v[a], j);
              at(out, j) = m * (1.0f / (float)na);
            }
          }
        }
        auto update = [&](int a, const float4& cfv) {
          float4 x = cell(a);
#pragma unroll
          for (int j = 0; j < VEC; j++) {
            const float y = at(x, j), disc = y > 0.0f ? d.pos : d.neg;
            at(x, j) = y * disc + (&cfv.x)[j] - at(out, j);
          }
          return x;
        };
        if constexpr (COMP) {
          float rmax = 0.0f;
          if (valid) {
#pragma unroll
            for (int a = 0; a < MAXA; a++)
              if (a < na) {
                v[a] = update(a, v[a]);
                rmax = fmaxf(rmax, absmax4(v[a]));
              }
          }
          const float mx = block_max(rmax, phase);
          const float rinv = mx > 0.0f ? 32767.0f / mx : 0.0f;
          if (tid == 0) A.rscale[st[i].cards] = mx;
          if (!valid) continue;
#pragma unroll
          for (int a = 0; a < MAXA; a++)
            if (a < na) {
              short4 q = make_short4(0, 0, 0, 0);
              if (mx > 0.0f)
                q = make_short4(enc_regret(v[a].x, rinv), enc_regret(v[a].y, rinv), enc_regret(v[a].z, rinv),
                                enc_regret(v[a].w, rinv));
              *reinterpret_cast<short4*>(A.rq + st[i].store + (size_t)(a * hp) + h0) = q;
            }
        } else {
          if (!valid) continue;
#pragma unroll
          for (int a = 0; a < MAXA; a++)
            if (a < na) st4(A.regrets + st[i].store + (size_t)(a * hp) + h0, update(a, v[a]));
        }
      }
    }
    st4(A.vals + (size_t)st[i].node * stride + h0, out);
  }
}

// A block's threads: one per 4 hands, whole warps.
unsigned threads_of(int hp) { return (unsigned)((hp + VEC * 32 - 1) / (VEC * 32) * 32); }

constexpr size_t SMEM_SM = 228 << 10, SMEM_BLOCK = 227 << 10, SMEM_STATIC = 4 << 10;  // static: with 1 KB reserved

// A stage: `rows` rows of 4 cells a thread. Where the segments are few, as much
// as leaves room for no more blocks on an SM than its share of them: blocks
// are placed while the kernel before drains, and the SMs that finish first
// would take most of them.
size_t stage_bytes(const RowArgs& A, int rows, int ntrees, int hp) {
  const size_t need = (size_t)rows * threads_of(hp) * (A.compressed ? 8 : 16);
  const size_t share = (size_t)(ntrees + A.sms - 1) / A.sms;
  return std::max(need, std::min(SMEM_SM / share, SMEM_BLOCK) - std::min(SMEM_SM / share, SMEM_STATIC));
}

template <int MODE, bool COMP>
auto down_kernel_for(int maxa) {
  return maxa <= 4   ? fused_down_kernel<MODE, 4, COMP>
         : maxa <= 8 ? fused_down_kernel<MODE, 8, COMP>
                     : fused_down_kernel<MODE, MAX_ACTIONS, COMP>;
}

template <int MODE, bool COMP>
auto up_kernel_for(int maxa) {
  return maxa <= 4   ? fused_up_kernel<MODE, 4, COMP>
         : maxa <= 8 ? fused_up_kernel<MODE, 8, COMP>
                     : fused_up_kernel<MODE, MAX_ACTIONS, COMP>;
}

template <int MODE>
void launch_down_mode(int maxa, const RowArgs& A, const FusedTree* trees, int ntrees, const DownTask* tasks, int hp,
                      cudaStream_t s) {
  const size_t smem = stage_bytes(A, (MODE == M_CFR ? 2 : 1) * maxa, ntrees, hp);
  launch_dependent(A.compressed ? down_kernel_for<MODE, true>(maxa) : down_kernel_for<MODE, false>(maxa),
                   dim3((unsigned)ntrees), threads_of(hp), smem, s, A, trees, tasks, maxa);
}

template <int MODE>
void launch_up_mode(int maxa, const RowArgs& A, const FusedTree* trees, int ntrees, const UpTask* tasks, int hp,
                    cudaStream_t s) {
  const size_t smem = stage_bytes(A, MODE == M_BR ? 0 : 2 * maxa, ntrees, hp);
  launch_dependent(A.compressed ? up_kernel_for<MODE, true>(maxa) : up_kernel_for<MODE, false>(maxa),
                   dim3((unsigned)ntrees), threads_of(hp), smem, s, A, trees, tasks, maxa);
}

template <int MODE>
cudaError_t allow(int bytes) {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto k) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  };
  for (int maxa : {4, 8, 16}) {
    set(down_kernel_for<MODE, false>(maxa));
    set(down_kernel_for<MODE, true>(maxa));
    set(up_kernel_for<MODE, false>(maxa));
    set(up_kernel_for<MODE, true>(maxa));
  }
  return e;
}

}  // namespace

cudaError_t fused_setup() {
  constexpr int most = (int)(SMEM_BLOCK - SMEM_STATIC);
  cudaError_t e = allow<M_CFR>(most);
  if (e == cudaSuccess) e = allow<M_BR>(most);
  if (e == cudaSuccess) e = allow<M_AVG>(most);
  return e;
}

void launch_fused_down(int mode, int maxa, const RowArgs& A, const FusedTree* trees, int ntrees,
                       const DownTask* tasks, int hp, cudaStream_t s) {
  if (ntrees <= 0) return;
  if (mode == M_CFR) launch_down_mode<M_CFR>(maxa, A, trees, ntrees, tasks, hp, s);
  else if (mode == M_BR) launch_down_mode<M_BR>(maxa, A, trees, ntrees, tasks, hp, s);
  else launch_down_mode<M_AVG>(maxa, A, trees, ntrees, tasks, hp, s);
}

void launch_fused_up(int mode, int maxa, const RowArgs& A, const FusedTree* trees, int ntrees, const UpTask* tasks,
                     int hp, cudaStream_t s) {
  if (ntrees <= 0) return;
  if (mode == M_CFR) launch_up_mode<M_CFR>(maxa, A, trees, ntrees, tasks, hp, s);
  else if (mode == M_BR) launch_up_mode<M_BR>(maxa, A, trees, ntrees, tasks, hp, s);
  else launch_up_mode<M_AVG>(maxa, A, trees, ntrees, tasks, hp, s);
}

}  // namespace dcfr
