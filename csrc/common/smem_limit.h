// A kernel's limit of dynamic shared memory belongs to the device that is current when it is raised, so a launcher that raises it
// once remembers on which devices it has.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace dptb {

// One per kernel (a static of its launcher).  Devices from 64 on are not remembered: the limit is raised at every launch.
struct SmemLimit {
  std::atomic<unsigned long long> raised{0};

  cudaError_t raise(const void* kernel, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (raised.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) raised.fetch_or(bit, std::memory_order_relaxed);
    return e;
  }
};

}  // namespace dptb
