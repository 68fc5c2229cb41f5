// esr_per_device.h -- work done once per device of the process.
#pragma once
#include <stdint.h>

#include <atomic>

namespace esr {

// A kernel's dynamic shared-memory limit belongs to the device that was
// current when it was raised, not to the process: a flag set on the first
// device would leave a launch on the second without it. `device` is marked once
// set(device) has returned 0; a failure is tried again by the next call. Safe
// from several threads (set() may then run more than once). Devices beyond 63
// are set on every call.
class PerDevice {
 public:
  template <typename Set>
  int once(int device, Set&& set) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = set(device);
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace esr
