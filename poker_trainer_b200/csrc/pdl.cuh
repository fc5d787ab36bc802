// Programmatic dependent launch: a kernel launched with launch_dependent may
// start once every block of the kernel before it has called pdl_trigger (or
// exited), and reads what earlier kernels wrote only after pdl_wait, which
// returns when that kernel is complete and its writes are visible.
#pragma once

#include <cuda_runtime.h>

namespace dcfr {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" :::); }

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
