// A setting that a device keeps per process and that is only ever raised (the
// shared-memory limit of a kernel): the largest value set so far on each device,
// so that a second device of the process gets it too.
#pragma once

#include <atomic>
#include <cstddef>

namespace gx {

class PerDevice {
public:
    // true when `value` has yet to be set on `device`
    bool needs(int device, size_t value) const {
        return device < 0 || device >= kDevices || set_[device].load(std::memory_order_acquire) < value;
    }
    void done(int device, size_t value) {
        if (device < 0 || device >= kDevices) return;  // (beyond the table: set at every launch)
        size_t old = set_[device].load(std::memory_order_relaxed);
        while (old < value && !set_[device].compare_exchange_weak(old, value, std::memory_order_release)) {
        }
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<size_t> set_[kDevices] = {};
};

}  // namespace gx
