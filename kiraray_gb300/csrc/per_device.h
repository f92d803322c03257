// What holds for a device and not for the process.
#pragma once

#include <atomic>
#include <cstdint>

namespace krr {

// Calls `set` until it has succeeded once on device `dev` (0 on success), and
// not again there; devices from 64 on call it every time.  Two threads may
// both call it: `set` gives the same state however often it runs.  Setting a
// kernel's shared-memory limit at every launch took 1 us of host time of a
// 13 us query.
class OncePerDevice {
  public:
    template <typename F>
    int operator()(int dev, F &&set) {
        const bool known = dev >= 0 && dev < 64;
        const uint64_t bit = known ? uint64_t(1) << dev : 0;
        if (known && (done_.load(std::memory_order_acquire) & bit)) return 0;
        const int status = set();
        if (status == 0 && known) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

  private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace krr
