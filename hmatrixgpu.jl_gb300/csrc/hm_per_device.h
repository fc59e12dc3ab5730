// Work to be done once per device of a process, such as raising a kernel's shared-memory
// limit, which holds for the device that is current when it is set. A static object of this
// class per such work; a failure is returned and tried again by the next call. Two threads
// that come first at once both do the work.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace hm {

class PerDevice {
  std::atomic<uint64_t> done{0};  // bit d: device d (later ones do the work every time)

 public:
  template <typename F>
  cudaError_t operator()(F work) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t(1) << dev : 0;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = work();
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

}  // namespace hm
