// Something that a process does once for every device it uses (a kernel's attributes belong to a device's copy of it).
#pragma once

#include <atomic>

class OncePerDevice {
public:
    // make() for the first call on this device, until it has returned 0; its result otherwise.
    template <typename F>
    int run(int device, F&& make) {
        const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0;      // (no bit: every time)
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int status = make();
        if (status == 0) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

private:
    std::atomic<unsigned long long> done_{0};
};
