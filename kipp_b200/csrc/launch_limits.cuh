// What a process has asked of each device for each kernel: how much dynamic shared memory its launches may take.  The
// limit belongs to a device, a launch above it is refused, and setting a smaller one takes the larger away; so it is kept
// per (device, kernel), raised under a lock and never lowered.  Plain C++.
#pragma once
#include <stddef.h>
#include <map>
#include <mutex>
#include <utility>

class SmemLimits {
public:
    static constexpr size_t WITHOUT_ASKING = 48 * 1024;
    // Sees to it that `kernel` may be launched with `bytes` on `device`: `set(bytes)` (0: done) where it may not yet.
    // Returns 0 or what `set` returned, which is asked again the next time.
    template <typename Set> int raise(int device, const void* kernel, size_t bytes, Set set) {
        if (bytes <= WITHOUT_ASKING) return 0;
        std::lock_guard<std::mutex> hold(mutex_);
        size_t& allowed = allowed_[std::make_pair(device, kernel)];
        if (bytes <= allowed) return 0;
        const int rc = set(bytes);
        if (rc == 0) allowed = bytes;
        return rc;
    }

private:
    std::mutex mutex_;
    std::map<std::pair<int, const void*>, size_t> allowed_;
};
