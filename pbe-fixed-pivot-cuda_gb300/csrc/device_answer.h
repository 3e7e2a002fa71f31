// =============================================================================
// device_answer.h -- a question about the current device, asked once on each.
// =============================================================================
#pragma once

#include <atomic>

namespace pbe_gb300 {

// What a kernel may do on a device (and the function attributes set to find out)
// belongs to that device alone: a process that works on several asks on every one.
// `ask` returns 1 (yes), -1 (no) or 0 (could not be found out: asked again next time).
// Threads may ask side by side: the answer is the same.
class DeviceAnswer {
public:
    static constexpr int kDevices = 64;
    template <class Ask>
    bool get(int device, Ask ask)
    {
        if (device < 0 || device >= kDevices) return ask() > 0;
        int a = known_[device].load(std::memory_order_acquire);
        if (a == 0) {
            a = ask();
            if (a != 0) known_[device].store(static_cast<signed char>(a), std::memory_order_release);
        }
        return a > 0;
    }

private:
    std::atomic<signed char> known_[kDevices] = {};
};

} // namespace pbe_gb300
