// What the CUDA runtime keeps per device (a kernel's shared-memory limit, how many of its clusters fit, a size of the device) is asked
// for or set once on each device that a process uses, not once per process.
#pragma once
#include <atomic>

namespace ib {

class PerDevice {
    static constexpr int MAX_DEVICES = 64;
    std::atomic<int> kept[MAX_DEVICES] = {};

public:
    // make()'s answer for this device. A positive one is kept (two threads that ask at once both make it: it is the same); any other
    // stands for a failure, which the next call tries again.
    template <typename F>
    int get(int device, F&& make) {
        if (device < 0 || device >= MAX_DEVICES) return make();
        int v = kept[device].load(std::memory_order_acquire);
        if (v <= 0) {
            v = make();
            if (v > 0) kept[device].store(v, std::memory_order_release);
        }
        return v;
    }
};

}  // namespace ib
