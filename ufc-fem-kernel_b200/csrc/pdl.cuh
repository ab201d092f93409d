// Programmatic dependent launch: the device-side entry of a kernel in a chain
// and its launcher.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace ufc {
namespace {

// Programmatic dependent launch between the kernels of a chain: each kernel waits
// for its predecessor's completion and memory (wait), then lets its successor
// launch as soon as all of its own blocks are running (launch_dependents); both
// are no-ops for a kernel launched without the attribute.  Before the wait a
// kernel may read only what its direct predecessor does not write: the matrix,
// flags, and vectors of earlier kernels.  Those are complete, because every
// kernel of a chain waits before it triggers its dependents, so the
// predecessor's own wait has seen them done; a kernel that triggered first, or
// left out the wait, would break that for the one after next.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
}

template <typename... K, typename... A>
void launch_pdl_smem(void (*kernel)(K...), int grid, int block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

template <typename... K, typename... A>
void launch_pdl(void (*kernel)(K...), int grid, int block, cudaStream_t st, A&&... args) {
  launch_pdl_smem(kernel, grid, block, 0, st, std::forward<A>(args)...);
}

}  // namespace
}  // namespace ufc
