// Programmatic dependent launch, shared by the product kernels: a kernel of a
// product may start while the one before it ends. It calls pdl_wait() before it
// touches anything that earlier kernels write (or still read), which returns when
// they are complete, and then pdl_trigger(), from which the next may start. What earlier
// kernels write (x too: it may be the y of the product before) changes while the kernel is
// already running, so it is not read through the read-only path: no __ldg, and no
// __restrict__ from which the compiler would take it to be constant or move a load up.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace hm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether the kernels of a pass of `columns` right-hand sides over `entries` stored entries may
// overlap: always in FP32. The CTAs of a kernel that starts while another ends land where there is
// room, several on one SM while others get none; that is made good where memory bounds the
// kernel, but not the FP64 pipe of the SMs. So in FP64 only while the launches are a good part of the
// time. Product in us with / without overlap, one column: 1000-point cube (0.99 M entries) 14.1 / 18.5,
// film of 3000 (2.7 M) 19.6 / 21.7, 1800-point cube (2.88 M) 23.1 / 24.6, sphere of 2500 (3.00 M) 31.9 / 23.6,
// 2500-point cube (5.0 M) 49.8 / 32.1; passes 4 to 32 wide, entries times width: 22 M 93.0 / 98.4, 29 M 79.5 /
// 85.9, 43 M 179.7 / 129.1 and 123.0 / 127.1, 81 M 341 / 219.
inline bool may_overlap(bool f64, int64_t entries, int columns) {
  return !f64 || entries * columns < (columns == 1 ? 2900000 : 30000000);
}

// A launch that may overlap the end of the kernel before it (`overlap`).
template <typename... P, typename... A>
static cudaError_t launch_pdl(bool overlap, void (*k)(P...), dim3 grid, int block, size_t smem, cudaStream_t s,
                              const A &...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(static_cast<unsigned>(block));
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

// The next unit of a CTA or warp, of n units shared by `workers` that began with the unit of their
// own number. Drawn when the unit before is done: drawn at its start, the first CTAs, which have the
// longest units, took the few that were left over (product of the 20,000-point cube at 1e-6, 1250 row
// units for 912 CTAs: FP32 191 us drawn early, 166 late; FP64 460 and 414; 32 FP64 columns of a
// 20,011-point sphere 3518 and 3130). No ticket where every unit has a worker.
__device__ __forceinline__ int32_t next_unit(int32_t *ticket, int32_t workers, int32_t n) {
  return n > workers ? workers + atomicAdd(ticket, 1) : n;
}

}  // namespace hm
