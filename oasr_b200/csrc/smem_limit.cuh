// A kernel's limit of dynamic shared memory, raised once on every device that launches it: the limit belongs to the device, so
// a flag for the whole process would leave the kernel unable to launch on a second one.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

namespace ob {

// One per kernel, as a static of its launcher.  Threads that meet here set the same limit twice, which is harmless.
class SmemLimit {
 public:
  template <typename Kernel>
  cudaError_t raise(Kernel kern, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t(1) << dev : 0;   // further devices: set on every launch
    if (raised_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kern), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) raised_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> raised_{0};
};

}  // namespace ob
