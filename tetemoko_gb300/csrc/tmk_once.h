// tmk_once.h -- settings of a device that a process makes once for each.
#pragma once
#include <atomic>

namespace tmk {

// A kernel's dynamic shared memory limit belongs to the current device, and a
// process may step on several: `set` (an error code, 0 for success) runs on the
// first call for each device and again on every call until it has succeeded.
// Threads that meet here first may each run it.
class DeviceOnce {
 public:
  template <typename Set> auto operator()(int device, Set&& set) -> decltype(set()) {
    const bool kept = device >= 0 && device < 64;
    const unsigned long long bit = kept ? 1ull << device : 0ull;
    if (done_.load(std::memory_order_acquire) & bit) return decltype(set())();
    const auto e = set();
    if (e == decltype(set())()) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<unsigned long long> done_{0};
};

}  // namespace tmk
