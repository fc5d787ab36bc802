// Programmatic dependent launch: a kernel launched with launch_dependent may
// start once every block of the kernel before it has called pdl_trigger (or
// exited), and reads what earlier kernels wrote only after pdl_wait, which
// returns when that kernel is complete and its writes are visible.
#pragma once

#include <cuda_runtime.h>

#include "plan.hpp"

namespace dcfr {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// PassTurn's work, by the first `blocks` blocks (those with tasks) of a
// terminal kernel, after their wait.
__device__ __forceinline__ void turn_pass(const PassTurn& T, uint32_t blocks = 1) {
  if (blockIdx.x >= blocks) return;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < T.nclear; i += blocks * blockDim.x) T.clear[i] = 0u;
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  if (T.step == TURN_NEXT) {
    const uint32_t t = *T.counter + 1;
    T.cur[1] = T.table[t < T.table_len ? t : T.table_len - 1];
  } else if (T.step == TURN_BEGIN) {
    *T.counter += 1;
    T.cur[0] = T.cur[1];
  }
}

template <typename... P, typename... A>
inline void launch_dependent(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t s,
                             A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace dcfr
