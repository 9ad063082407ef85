// A kernel's limit of dynamic shared memory: raised on each device that launches it (a function's attributes are those of one device), and there to
// the largest size asked for. One static object per kernel; safe with several threads.
#pragma once
#include <cuda_runtime_api.h>
#include <atomic>
#include <mutex>

namespace qspec {

class SmemLimit {
 public:
  template <typename Kernel>
  cudaError_t raise(Kernel kernel, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool known = dev < DEVICES;
    if (known && (size_t)raised_[dev].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
    std::lock_guard<std::mutex> lock(mutex_);            // two sizes at once: the larger one stays
    if (known && (size_t)raised_[dev].load(std::memory_order_relaxed) >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && known) raised_[dev].store((int)bytes, std::memory_order_release);
    return e;
  }

 private:
  static constexpr int DEVICES = 64;
  std::atomic<int> raised_[DEVICES] = {};
  std::mutex mutex_;
};

}  // namespace qspec
