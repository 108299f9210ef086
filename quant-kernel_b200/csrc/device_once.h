// device_once.h -- set-up that belongs to a device, done once for each.
//
// cudaFuncSetAttribute and the like apply to the current device only: a flag of
// the process would leave the second GPU of a program without them.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace qkb {

class DeviceOnce {
public:
    static constexpr int kDevices = 64;
    // setup() for `device` unless it has succeeded before; its result, 0 being
    // success.  A failure is not kept.
    template <class Setup>
    auto run(int device, const Setup& setup) -> decltype(setup()) {
        using Result = decltype(setup());
        if (device < 0 || device >= kDevices) return setup();
        const uint64_t bit = uint64_t{1} << device;
        if (done_.load(std::memory_order_acquire) & bit) return Result{};
        std::lock_guard<std::mutex> lock(mu_);
        if (done_.load(std::memory_order_relaxed) & bit) return Result{};
        const Result r = setup();
        if (r == Result{}) done_.fetch_or(bit, std::memory_order_release);
        return r;
    }

private:
    std::atomic<uint64_t> done_{0};
    std::mutex mu_;
};

}  // namespace qkb
