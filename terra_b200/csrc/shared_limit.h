// The limit of a kernel's dynamic shared memory beyond the 48 KB that every launch may have. It belongs to the kernel and the device, so it is
// raised at the first launch on each device.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>

namespace tb {

class SharedLimit {
 public:
  // `bytes`: the most that the kernel is ever launched with, always the same (a thread's lower limit would undo another's)
  cudaError_t raise(const void* kernel, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
    if (devices_.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) devices_.fetch_or(bit, std::memory_order_relaxed);
    return e;
  }

 private:
  std::atomic<unsigned long long> devices_{0};      // a bit per device (beyond 64 of them the call is made each time)
};

}  // namespace tb
