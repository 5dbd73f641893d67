// lmb_smem.h -- a kernel's dynamic shared-memory limit, raised as launches
// need it.
#pragma once

#include <stddef.h>

#include <atomic>
#include <mutex>

namespace lmb {

// Raised once per device to the largest size asked for so far (setting it on
// every launch costs host time comparable to a small kernel) and never
// lowered: threads that launch with different sizes at the same time set it
// one after another, each only above what is granted.  set(bytes) sets the
// limit on the current device and returns 0 when it could.
class SmemLimit {
public:
    static constexpr int DEVICES = 64;
    static constexpr int BAD_DEVICE = -1;

    template <class Set>
    int raise(int device, size_t bytes, Set set)
    {
        if (device < 0 || device >= DEVICES) return BAD_DEVICE;
        std::atomic<size_t> &g = granted_[device];
        if (bytes <= g.load(std::memory_order_acquire)) return 0;
        std::lock_guard<std::mutex> lock(mutex_);
        if (bytes <= g.load(std::memory_order_relaxed)) return 0;
        const int rc = set(bytes);
        if (rc == 0) g.store(bytes, std::memory_order_release);
        return rc;
    }

private:
    std::mutex mutex_;
    std::atomic<size_t> granted_[DEVICES] = {};
};

}  // namespace lmb
