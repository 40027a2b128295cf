// An answer that is found once per device: what a device can launch, after the
// kernel attributes it needs were set on it (they belong to a function on a device,
// so an answer of the first device says nothing about a second one).
#pragma once

#include <mutex>

namespace moea {

class PerDevice {
public:
    // The answer of `probe()` (bool) on `device`, the current device; found on the
    // first call for it, by one thread while others wait.  Devices past the table
    // are probed on every call.
    template <class Probe>
    bool get(int device, Probe probe)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        if (device < 0 || device >= kDevices) return probe();
        if (answer_[device] == 0) answer_[device] = probe() ? 1 : -1;
        return answer_[device] > 0;
    }

private:
    static constexpr int kDevices = 64;
    std::mutex mutex_;
    signed char answer_[kDevices] = {};  // 0 unknown, 1 yes, -1 no
};

}  // namespace moea
