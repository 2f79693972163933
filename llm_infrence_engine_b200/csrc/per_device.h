// What has to be done once for every device of a process (a kernel's room in shared memory, for one), whichever threads and devices
// come first. Plain C++: the caller brings the device and the call.
#pragma once

#include <stdint.h>

#include <atomic>

class OncePerDevice {
    std::atomic<uint64_t> done_{0};   // a bit per device; devices from 64 on are asked every time

public:
    // Runs `what` unless it has succeeded (returned 0) for this device before. Two threads may both run it, a failure is tried again.
    template <typename What> int run(int device, What what) {
        const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int rc = what();
        if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
        return rc;
    }
};
