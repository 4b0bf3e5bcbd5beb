// What a kernel needs set before it is launched: dynamic shared memory beyond 48 KB, and all of the
// unified L1/shared storage as shared memory where two of its CTAs are to fit on an SM. A setting holds on
// the device that is current when it is made, so it is made once per kernel and device, by the first launch
// there (not a stream operation: a first launch inside a stream capture is fine).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace shz {

class LaunchAttr {
 public:
  // Called ahead of each launch of k, on the device it is launched on. Launches of several threads may
  // set the same values side by side; a setting that fails is tried again by the next launch.
  cudaError_t set(const void* k, size_t shared_bytes, bool carveout) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool kept = dev >= 0 && dev < 64;  // (beyond: set ahead of every launch)
    if (kept && ((done_.load(std::memory_order_acquire) >> dev) & 1u)) return cudaSuccess;
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared_bytes);
    if (e == cudaSuccess && carveout)
      e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess && kept) done_.fetch_or(1ull << dev, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};  // bit d: set on device d
};

}  // namespace shz
