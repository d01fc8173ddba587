// Facts of the current device that launchers size their grids by.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace moloch {

// SMs of the current device, looked up once on each (safe with several
// threads: all of them find the same number)
inline int sm_count() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  const bool cached = dev >= 0 && dev < 64;
  int n = cached ? known[dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 1;
  if (cached) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace moloch
