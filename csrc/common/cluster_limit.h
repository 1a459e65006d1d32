// How many clusters of a kernel can be resident at once on the current device: asked once per device.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "common/smem_limit.h"

namespace dptb {

// One per kernel and cluster size (a static of its launcher).  Devices from 64 on are asked at every launch.
struct ClusterLimit {
  // 0 when the question fails.  It is then put again at the next launch, and no error stays behind that an ordinary launch after it
  // would take for its own.
  int resident(const void* kernel, SmemLimit& smem, int smem_bytes, const cudaLaunchConfig_t& cfg) {
    int dev = 0, n = 0;
    cudaError_t e = cudaGetDevice(&dev);
    const bool kept = e == cudaSuccess && dev < 64;
    if (kept && (n = counts[dev].load(std::memory_order_relaxed)) > 0) return n - 1;
    if (e == cudaSuccess) e = smem.raise(kernel, smem_bytes);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    if (kept) counts[dev].store(n + 1, std::memory_order_relaxed);
    return n;
  }

 private:
  std::atomic<int> counts[64]{};      // one more than the number; 0: not asked for yet
};

}  // namespace dptb
