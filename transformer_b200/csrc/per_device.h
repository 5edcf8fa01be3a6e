// Something that has to be done once on every device that a process uses: a kernel's limits, for instance, are kept by the
// runtime per device.
#pragma once
#include <atomic>

class PerDevice {
    std::atomic<unsigned long long> done_{0};

public:
    // `act` (true: it went well) unless it has gone well on `device` before.  Threads may call it side by side: `act` may then
    // run more than once.  Devices from 64 on are not remembered.
    template <typename Act> void once(int device, Act act) {
        const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0;
        if (bit && (done_.load(std::memory_order_acquire) & bit)) return;
        if (act()) done_.fetch_or(bit, std::memory_order_release);
    }
};
