// Whole numbers that cost models ask the runtime for once per device.
#pragma once
#include <atomic>

// KEYS positive numbers for each of 64 devices.  Threads that ask for the same one at once may each ask the runtime, and keep the same answer.
template <int KEYS>
class DeviceTable {
    static constexpr int DEVICES = 64;
    std::atomic<int> known_[DEVICES][KEYS] = {};

public:
    // What ask() said for this device and key; it is asked again where it said 0 or less (no answer), or the device is beyond the table
    template <class Ask>
    int get(int device, int key, Ask ask) {
        const bool kept = device >= 0 && device < DEVICES && key >= 0 && key < KEYS;
        if (kept) {
            const int n = known_[device][key].load(std::memory_order_relaxed);
            if (n > 0) return n;
        }
        const int n = ask();
        if (kept && n > 0) known_[device][key].store(n, std::memory_order_relaxed);
        return n;
    }
};
