// What a process asks for once per device.  A kernel's attributes belong to the device's copy of the kernel, and a process may run
// engines on several devices: what one of them granted says nothing of the next.  Plain C++, without CUDA.
#pragma once
#include <atomic>
#include <mutex>
#include <stddef.h>

#define RB_MAX_DEVICES 64

// A static object (all zeros at the start), usable from any number of threads.
struct RbPerDevice {
    std::atomic<size_t> granted[RB_MAX_DEVICES];
    std::mutex mu;
    // set() grants `want`; it is called unless that much has been granted on `dev` before.  Returns 0, or what set() returned: then
    // nothing counts as granted, and the next call tries again.
    template <typename Set> int raise(int dev, size_t want, Set&& set) {
        if (dev < 0 || dev >= RB_MAX_DEVICES) return set();
        if (granted[dev].load(std::memory_order_acquire) >= want) return 0;
        std::lock_guard<std::mutex> g(mu);
        if (granted[dev].load(std::memory_order_relaxed) >= want) return 0;
        const int e = set();
        if (e == 0) granted[dev].store(want, std::memory_order_release);
        return e;
    }
};
