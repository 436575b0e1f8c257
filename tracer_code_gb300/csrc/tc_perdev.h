// Values that belong to a device (SM counts, what fits it) and settings made once for each
// (kernel attributes).  A process may hold handles on several devices.
#pragma once
#include <atomic>

int tc_current_device();  // the calling thread's

class PerDevice {
public:
    // f() of the current device: f is called until it returned a value that is not
    // negative, then that value is kept (f may run more than once when threads race)
    template <class F>
    int get(F f) {
        const int dev = tc_current_device();
        if (dev < 0 || dev >= kDevices) return f();
        int v = kept[dev].load(std::memory_order_acquire);
        if (v == 0) {
            v = f() + 1;
            if (v <= 0) return v - 1;
            kept[dev].store(v, std::memory_order_release);
        }
        return v - 1;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<int> kept[kDevices] = {};  // value + 1; 0: not known
};

int tc_sm_count();  // SMs of the current device
