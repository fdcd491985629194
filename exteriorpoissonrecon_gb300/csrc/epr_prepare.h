// Once-per-device preparation (tables and attributes of the kernels), made by the first context on a device.
#pragma once
#include <map>
#include <mutex>

namespace epr {

template <typename T>
class PerDevice
{
    std::mutex mutex_;
    std::map<int, T> made_;

public:
    // out = the device's T, made by make(T &) the first time; where make returns false nothing is kept, so that
    // the next call tries again, and the result is false
    template <typename F>
    bool get(int device, T &out, F &&make)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        auto at = made_.find(device);
        if (at == made_.end())
        {
            T t{};
            if (!make(t)) return false;
            at = made_.emplace(device, t).first;
        }
        out = at->second;
        return true;
    }
};

}  // namespace epr
