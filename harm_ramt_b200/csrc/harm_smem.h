// The dynamic shared memory limit of a kernel that asks for more than 48 KB.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace harm {

// Raises a kernel's limit at its first launch on each device: the limit
// belongs to the device's copy of the kernel, so one raised for the first
// device of a process would leave the launches on a second one refused.
struct SmemLimit {
  std::atomic<uint64_t> done{0};  // a bit for each of the first 64 devices
  void raise(const void* kern, size_t bytes)
  {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    const uint64_t bit = (dev < 64) ? uint64_t(1) << dev : 0;
    if (done.load(std::memory_order_relaxed) & bit) return;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
      done.fetch_or(bit, std::memory_order_relaxed);
  }
};

}  // namespace harm
