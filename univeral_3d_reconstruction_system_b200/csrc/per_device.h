// per_device.h - values that belong to a device rather than to the process (plain C++).
//
// A function attribute (the shared memory that a kernel may use) is set on the current device's copy of the
// kernel, and an occupancy is the current device's, so a launcher asks once per device. Callers may be on
// several threads: two may compute the value at the same time, which gives the same result.
#pragma once

#include <atomic>

namespace u3dg {

class PerDevice {
  public:
    // The device's value: make(), not 0, on the first call for the device.
    template <class F>
    int get(int device, F &&make)
    {
        if (device < 0 || device >= kDevices)
            return make();
        int v = values[device].load(std::memory_order_acquire);
        if (v == 0) {
            v = make();
            values[device].store(v, std::memory_order_release);
        }
        return v;
    }

  private:
    static constexpr int kDevices = 64;
    std::atomic<int> values[kDevices] = {};
};

} // namespace u3dg
