// Raising a kernel's dynamic shared-memory limit once per device.  The limit is
// an attribute of the function on one device: a process that opens several has
// to set it on each.
#pragma once

#include <atomic>

namespace dk {

class SmemLimit {
  public:
    // Calls `set()` (0: done) unless it has succeeded for `device` before; returns its result.  Threads may both call
    // it: it always sets the same size.  Device ordinals beyond the table set it every time.
    template <class Set>
    int raise(int device, Set set) {
        const bool kept = device >= 0 && device < kDevices;
        if (kept && done_[device].load(std::memory_order_acquire)) return 0;
        const int error = (int)set();
        if (kept && error == 0) done_[device].store(true, std::memory_order_release);
        return error;
    }

  private:
    static constexpr int kDevices = 64;
    std::atomic<bool> done_[kDevices] = {};
};

}  // namespace dk
