// Set-up that belongs to a device and not to the process: kernel function attributes (cudaFuncSetAttribute applies to the current
// device only, and contexts of several devices may live in one process).
#pragma once
#include <mutex>
#include <set>

namespace enn_b200 {

// Runs `set` (called with `device` current; returns 0 on success) once for each device.  A failure is returned and not remembered: the
// next call tries again.
class PerDeviceInit {
  public:
    template <typename F>
    auto run(int device, F set) -> decltype(set()) {
        std::lock_guard<std::mutex> lock(mutex_);
        if (done_.count(device)) return decltype(set())();
        const auto e = set();
        if (e == decltype(set())()) done_.insert(device);
        return e;
    }

  private:
    std::mutex mutex_;
    std::set<int> done_;
};

}  // namespace enn_b200
