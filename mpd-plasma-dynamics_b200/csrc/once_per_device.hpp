// Work to be done once on every GPU that a process uses, from any thread (a
// function attribute belongs to the current device's copy of the function).
#pragma once

#include <atomic>

namespace mpd {

class OncePerDevice {
public:
    // Runs set() unless it has already returned 0 on this device; returns what
    // it returned.  Threads that meet here for the first time may all run it.
    template <class Set>
    int operator()(int device, Set set) {
        const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int rc = static_cast<int>(set());
        if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
        return rc;
    }

private:
    std::atomic<unsigned long long> done_{0};
};

}  // namespace mpd
