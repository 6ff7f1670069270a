// What a launcher keeps per device: attributes of a kernel belong to a (kernel, device) pair, and launchers are called from
// several host threads (different handles may be used from different threads).  No CUDA in here, so that it can be tested
// with stand-ins for the calls.
#pragma once
#include <atomic>
#include <cstddef>
#include <mutex>

namespace wick {

constexpr int MAX_DEVICES = 64;  // devices beyond it are served without the memory: every call sets the value again

// A limit that is only ever raised: a caller with a smaller need must not lower it under one that is about to launch with a
// larger one.  `set(value)` runs under the lock and returns 0 (success) or an error code, which is passed on; the fast path is
// one atomic load.  One static object per kernel.
class RaisedPerDevice {
    std::mutex lock;
    std::atomic<size_t> granted[MAX_DEVICES] = {};
    size_t beyond = 0;  // the largest request of the devices without a place of their own

public:
    template <class Set>
    int raise(int device, size_t value, Set&& set) {
        const bool known = device >= 0 && device < MAX_DEVICES;
        if (known && granted[device].load(std::memory_order_acquire) >= value) return 0;
        std::lock_guard<std::mutex> hold(lock);
        if (!known) {
            beyond = value > beyond ? value : beyond;
            return set(beyond);
        }
        if (granted[device].load(std::memory_order_relaxed) >= value) return 0;
        const int e = set(value);
        if (e == 0) granted[device].store(value, std::memory_order_release);
        return e;
    }
};

}  // namespace wick
