// Something a process does once for each of its devices, such as setting an attribute that belongs to the current device.
#pragma once
#include <atomic>

namespace adop {

class OncePerDevice
{
   public:
    static constexpr int kDevices = 64;  // beyond them it is done on every call
    // f() returns 0 when it has succeeded; until then it is called again. Threads that come at the same time may all call it.
    template <class F>
    auto run(int device, F f) -> decltype(f())
    {
        const bool known = device >= 0 && device < kDevices;
        if (known && done_[device].load(std::memory_order_acquire)) return decltype(f())(0);
        const auto r = f();
        if (known && r == decltype(f())(0)) done_[device].store(true, std::memory_order_release);
        return r;
    }

   private:
    std::atomic<bool> done_[kDevices] = {};
};

}  // namespace adop
