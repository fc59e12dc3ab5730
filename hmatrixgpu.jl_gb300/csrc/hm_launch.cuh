// Programmatic dependent launch, shared by the product kernels: a kernel of a
// product may start while the one before it ends. It calls pdl_wait() before it
// touches anything that earlier kernels write (or still read), which returns when
// they are complete, and then pdl_trigger(), from which the next may start.
#pragma once
#include <cuda_runtime.h>

namespace hm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
static cudaError_t launch_pdl(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(static_cast<unsigned>(grid));
  c.blockDim = dim3(static_cast<unsigned>(block));
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

}  // namespace hm
