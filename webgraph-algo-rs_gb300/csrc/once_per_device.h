// Settings that belong to a device and not to the process.
#pragma once
#include <atomic>
#include <cstdint>

namespace hbl {

// Runs `set` (0: success) on each device until it succeeded there once; a failure
// is returned and not kept. Safe with several threads, which may at worst run
// `set` once each.
class OncePerDevice {
    std::atomic<uint64_t> done_{0};

  public:
    template <class F>
    int operator()(int device, F&& set) {
        const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0;  // others: every time
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int e = set();
        if (e == 0) done_.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

}  // namespace hbl
