// Work that is done once for every device of the process, whichever thread comes first.
#pragma once
#include <atomic>
#include <cstdint>

struct PerDeviceOnce {
  std::atomic<uint64_t> done{0};
  // set() for this device unless it has succeeded (returned zero) before; devices beyond 63 call it
  // every time.
  template <class F> auto operator()(int device, F set) -> decltype(set()) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
    if (done.load(std::memory_order_acquire) & bit) return decltype(set())(0);
    const auto r = set();
    if (r == decltype(set())(0)) done.fetch_or(bit, std::memory_order_release);
    return r;
  }
};
