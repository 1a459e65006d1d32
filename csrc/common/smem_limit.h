// A kernel's limit of dynamic shared memory belongs to the device that is current when it is raised, so a launcher that raises it
// once remembers on which devices it has.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace dptb {

// One per kernel (a static of its launcher).  Devices from 64 on are not remembered: the limit is raised at every launch.
struct SmemLimit {
  cudaError_t raise(const void* kernel, int bytes) { return set(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }
  // Clusters of more than 8 CTAs (an object of its own beside the limit's).
  cudaError_t allow_wide_clusters(const void* kernel) { return set(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1); }

 private:
  cudaError_t set(const void* kernel, cudaFuncAttribute what, int value) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (raised.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, what, value);
    if (e == cudaSuccess) raised.fetch_or(bit, std::memory_order_relaxed);
    return e;
  }
  std::atomic<unsigned long long> raised{0};
};

}  // namespace dptb
