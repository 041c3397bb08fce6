// Once per device instead of once per process: what is set for a kernel (its dynamic shared memory, its cluster sizes) holds for the
// device that is current at the call, and a process may have contexts on several.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>

class RtDeviceOnce {
 public:
  // Calls `set` unless it has succeeded on this device already.  Threads that come first together both call it.
  template <class F>
  cudaError_t operator()(F set) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const uint64_t bit = device < 64 ? uint64_t(1) << device : 0;  // beyond: every time
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = set();
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};
