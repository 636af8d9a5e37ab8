// A kernel's opt-in to more than 48 KB of dynamic shared memory.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>

namespace msbg {

// The attribute belongs to a kernel on a device, so one object per kernel (a function-local
// static) keeps which of the process's devices have it.  Safe to call from several threads.
class SmemOptIn {
 public:
  cudaError_t operator()(const void *kernel, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;  // further devices: set on every call
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace msbg
