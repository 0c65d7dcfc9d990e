// A value that is computed once per device.
//
// Kernel attributes (the opt-in shared memory, non-portable clusters) belong to the
// device that is current when they are set, and so does the answer which cluster
// can be resident: a static that is set once per process leaves the kernel's launch
// on a second device without them.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <mutex>

namespace jfg {

class PerDevice {
public:
    // f() with the current device's value; called once per device, by one thread.
    // When it throws nothing is kept and the next call tries again.
    template <class F>
    int get(F&& f)
    {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return f();
        Slot& s = slot[dev];
        if (!s.have.load(std::memory_order_acquire)) {
            std::lock_guard<std::mutex> g(m);
            if (!s.have.load(std::memory_order_relaxed)) {
                s.value = f();
                s.have.store(true, std::memory_order_release);
            }
        }
        return s.value;
    }

private:
    static constexpr int kDevices = 64;
    struct Slot {
        std::atomic<bool> have{false};
        int value = 0;
    };
    Slot slot[kDevices];
    std::mutex m;
};

}  // namespace jfg
