// A kernel's attributes (its limit of shared memory, whether it may run in
// clusters of 16) belong to a device: set once on each, from whichever thread
// launches there first.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace lace {

// done(f): f() has succeeded on the calling thread's device (called there at the
// first call, and again while it fails)
class PerDevice {
 public:
  template <typename F>
  bool done(F f) {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) return false;
    const unsigned long long bit = d < 64 ? 1ull << d : 0;  // past 64 devices at every call
    if (set_.load(std::memory_order_relaxed) & bit) return true;
    if (!f()) return false;
    set_.fetch_or(bit, std::memory_order_relaxed);
    return true;
  }

 private:
  std::atomic<unsigned long long> set_{0};
};

}  // namespace lace
