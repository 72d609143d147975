// smem_allowed.h — a kernel's dynamic shared memory above 48 KB is allowed per
// device: a handle on a second device of the process needs it again.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>

namespace gprx {

// One object per kernel (a static of its launcher): sets the attribute at the
// kernel's first launch on each device.
class SmemAllowed {
 public:
  cudaError_t operator()(const void* kernel, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (devices_.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) devices_.fetch_or(bit, std::memory_order_relaxed);
    return e;
  }

 private:
  std::atomic<unsigned long long> devices_{0};
};

}  // namespace gprx
