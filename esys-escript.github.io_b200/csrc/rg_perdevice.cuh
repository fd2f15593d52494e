// Set-up that belongs to the device that is current when it is done (a kernel's attributes, a device's
// properties), once per device.  No CUDA in here: tests run it on the host.
#pragma once
#include <mutex>

namespace rg {

constexpr int kMaxDevices = 64;

class PerDevice {
    std::mutex mu_;
    bool done_[kMaxDevices] = {};

public:
    // set() unless it has returned `ok` for device `dev` before
    template <class E, class F>
    E run(int dev, E ok, F set)
    {
        if (dev < 0 || dev >= kMaxDevices) return set();
        std::lock_guard<std::mutex> lock(mu_);
        if (done_[dev]) return ok;
        const E e = set();
        done_[dev] = e == ok;
        return e;
    }
};

}  // namespace rg
