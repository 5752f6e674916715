// What a process does once per device: a kernel's attribute (its share of dynamic shared memory) belongs to the device that was current when it was
// set, so a launch that remembers it for the process fails on the second device.
#pragma once
#include <atomic>

struct VmOncePerDevice {
    // `f` (0: done) runs at the first call on each device, and again as long as it fails; several threads may run it at the same time.  Devices
    // from 64 on are not remembered.
    template <class F> int operator()(int device, F&& f) {
        const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int status = f();
        if (status == 0) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

private:
    std::atomic<unsigned long long> done_{0};
};
