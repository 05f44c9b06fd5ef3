// ib_optin.h -- the dynamic shared memory that a kernel has been opted in to, per device.
//
// The attribute belongs to a kernel on one device, and a later, smaller value lowers it again, so one number per
// process is not enough: a launch on a second device would fail, and two threads whose sizes differ could leave
// the smaller one set.
#pragma once

#include <atomic>
#include <cstddef>
#include <mutex>

namespace ib {

class SmemOptIn {
public:
    // Makes sure that at least `bytes` are set on `device`: set(bytes) sets the attribute there and returns 0, or a
    // status that is passed on and leaves the record as it was.
    template <typename Set>
    int raise(int device, size_t bytes, Set &&set)
    {
        const bool recorded = device >= 0 && device < kDevices;
        if (recorded && bytes <= have_[device].load(std::memory_order_acquire)) return 0;
        std::lock_guard<std::mutex> lock(mutex_);
        if (recorded && bytes <= have_[device].load(std::memory_order_relaxed)) return 0;
        const int rc = set(bytes);
        if (rc == 0 && recorded) have_[device].store(bytes, std::memory_order_release);
        return rc;
    }

private:
    static constexpr int kDevices = 32;
    std::atomic<size_t> have_[kDevices] = {};
    std::mutex mutex_;
};

}  // namespace ib
