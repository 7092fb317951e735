// Opt-in to more than 48 KB of dynamic shared memory, once per kernel and device.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace laker {

// One per kernel (a function-local static of its launcher).  The attribute belongs
// to the kernel on one device: a process may launch on several, from several
// threads, so what is remembered is a bit per device.  Setting it twice is harmless.
class SmemOptIn {
 public:
  // Allows `kernel` `bytes` of dynamic shared memory on the current device.
  template <typename Kernel>
  cudaError_t allow(Kernel* kernel, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t(1) << dev : 0;
    if (done_.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_relaxed);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace laker
