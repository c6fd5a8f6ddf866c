// psv_device.hpp -- what is set or asked once per GPU of a process.
#pragma once

#include <map>
#include <mutex>

namespace psv {

// A value for each device, made where it is first asked for (a kernel's
// attributes and occupancy are the device's that is current when they are set).
// Any number of threads may ask; one makes it.
template <typename V> class PerDevice {
    std::mutex m;
    std::map<int, V> made;

public:
    template <typename F> V get(int device, F make)
    {
        std::lock_guard<std::mutex> lock(m);
        auto it = made.find(device);
        if (it == made.end()) it = made.emplace(device, make()).first;
        return it->second;
    }
};

}  // namespace psv
