// tm_per_device.h -- a setup that has to be made once on each device.
//
// A kernel's attributes belong to a device (its context), and host threads with
// contexts of their own may launch the same kernel for the first time together: a
// plain "done" flag per process would leave the second device without the setup and
// race between the threads.  Host code only; no CUDA here, so the tests run it alone.
#pragma once
#include <atomic>

namespace tmg {

class PerDevice {
public:
    // setup() where no earlier one succeeded on this device; returns its error code (0:
    // success, what a repeated call returns too).  Two threads that come first together
    // both run it, so it must bear repeating.
    template <typename Setup>
    auto run(int device, Setup setup) -> decltype(setup())
    {
        const bool tracked = device >= 0 && device < 64;
        const unsigned long long bit = tracked ? 1ULL << device : 0ULL;
        if (tracked && (done_.load(std::memory_order_acquire) & bit)) return decltype(setup()){};
        const auto error = setup();
        if (tracked && error == decltype(setup()){}) done_.fetch_or(bit, std::memory_order_release);
        return error;
    }

private:
    std::atomic<unsigned long long> done_{0};
};

}  // namespace tmg
