// per_device.cuh -- something done once per device of the process (plain C++).
#pragma once

#include <atomic>
#include <mutex>

namespace att {

// run(device, f) calls f() the first time it is asked for a device and returns
// its status; later calls for that device return 0 without it.  A failure is
// returned and tried again by the next call.  Devices past kMax run f() every
// time.  Constant-initialised, so one can be a function's static.
class OncePerDevice {
public:
    static constexpr int kMax = 64;
    template <typename F>
    int run(int device, F f) {
        if (device < 0 || device >= kMax) return f();
        if (done_[device].load(std::memory_order_acquire)) return 0;
        std::lock_guard<std::mutex> lock(mutex_);
        if (done_[device].load(std::memory_order_relaxed)) return 0;
        const int status = f();
        if (status == 0) done_[device].store(true, std::memory_order_release);
        return status;
    }

private:
    std::atomic<bool> done_[kMax] = {};
    std::mutex mutex_;
};

}  // namespace att
