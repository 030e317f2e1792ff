// One-time set-up per CUDA device.
#pragma once
#include <atomic>
#include <cstdint>

namespace mpm {

// Runs a set-up step once for each device: a kernel's attributes (its limit of
// dynamic shared memory) belong to the device that was current when they were
// set, so one flag for the process leaves the second device without them.  Safe
// with several threads: two that meet on a device may both run the step, and
// neither returns before it has run.  A step that fails (does not return 0,
// cudaSuccess) is run again on the next call; devices past the 64th run it on
// every call.
class OncePerDevice {
public:
    template <class F>
    auto operator()(int device, F&& setup) -> decltype(setup()) {
        const uint64_t bit = device >= 0 && device < 64 ? (uint64_t)1 << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return {};
        const auto e = setup();
        if (e == decltype(e){}) done_.fetch_or(bit, std::memory_order_release);
        return e;
    }

private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace mpm
