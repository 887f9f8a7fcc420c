// Values a kernel's launches need once per device (an attribute set, an occupancy asked): kept per device, since
// function attributes belong to a device, and safe with several threads.
#pragma once

#include <atomic>
#include <cuda_runtime_api.h>

namespace tdg {

// The current device's value of a cache: positive once `make()` has given one there.  make() returns the
// value, or a value <= 0 on failure, which is not kept.  Two threads may both make it.
class PerDevice {
public:
    template <class Make>
    int get(Make&& make) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return 0;
        if (dev < 0 || dev >= kDevices) return make();
        int v = value_[dev].load(std::memory_order_acquire);
        if (v <= 0) {
            v = make();
            if (v > 0) value_[dev].store(v, std::memory_order_release);
        }
        return v;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<int> value_[kDevices] = {};
};

}  // namespace tdg
