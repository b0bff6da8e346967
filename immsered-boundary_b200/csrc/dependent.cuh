// Programmatic dependent launch of chains of kernels (the kernels of a time
// step, of a training step).
#pragma once

#include <cuda_runtime.h>

namespace ibgpu {

// A kernel of a chain lets the next one be set up as soon as all its CTAs run, and waits for the previous one to have
// completed before it reads or writes anything that the chain changes
// (tables that no kernel of a run writes may be read before).
__device__ __forceinline__ void dep_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void dep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// smem: bytes of dynamic shared memory
template <typename... P, typename... A>
void launch_dep_smem(bool dep, cudaStream_t st, dim3 grid, dim3 block, size_t smem,
                     void (*kernel)(P...), const A &...args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = dep ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
template <typename... P, typename... A>
void launch_dep(bool dep, cudaStream_t st, dim3 grid, dim3 block, void (*kernel)(P...),
                const A &...args) {
  launch_dep_smem(dep, st, grid, block, 0, kernel, args...);
}

}  // namespace ibgpu
