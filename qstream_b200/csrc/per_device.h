// A positive number that each device has its own of (how many blocks it runs at once), asked for once per device.  Any thread may be the first;
// no answer (0) is not remembered.
#pragma once

#include <atomic>

class PerDevice {
public:
    template <typename Ask>
    int get(int device, Ask ask) {
        const bool kept = device >= 0 && device < DEVICES;
        int n = kept ? known_[device].load(std::memory_order_acquire) : 0;
        if (n > 0) return n;
        n = ask();
        if (kept && n > 0) known_[device].store(n, std::memory_order_release);
        return n;
    }

private:
    static constexpr int DEVICES = 64;
    std::atomic<int> known_[DEVICES] = {};
};
