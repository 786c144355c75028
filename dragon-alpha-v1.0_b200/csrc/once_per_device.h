// What has to be set once for each device of a process.
#pragma once
#include <atomic>
#include <cstdint>

namespace alpha {

constexpr int kMaxDevices = 64;   // devices of a process that the library serves

// Runs a setup (0 = done) on each device until it has succeeded there once.  Threads that come together may both run it: a setup
// is one that may be repeated.
class OncePerDevice {
    std::atomic<uint64_t> done_{0};
public:
    template <class Setup>
    int operator()(int device, Setup setup)
    {
        if (device < 0 || device >= kMaxDevices) return setup();
        const uint64_t bit = uint64_t{1} << device;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int rc = setup();
        if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
        return rc;
    }
};

}  // namespace alpha
