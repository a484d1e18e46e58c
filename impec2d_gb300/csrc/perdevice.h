// Host-side state that exists once per device of a process (no CUDA types: also compiled alone by the tests).
#pragma once
#include <atomic>
#include <mutex>

namespace impec {

// Something each device needs once, such as a kernel's shared-memory limit: do_once(dev, ok, f) calls f until it has
// returned ok for that device.  Devices beyond the 64 that are remembered call f every time, which does
// no harm.  Safe with several threads: f runs under the lock, which later calls do not take.
class OncePerDevice {
    std::mutex mu;
    std::atomic<unsigned long long> done{0};

public:
    template <class R, class F>
    R do_once(int dev, R ok, F&& f) {
        const bool kept = dev >= 0 && dev < 64;
        if (kept && (done.load(std::memory_order_acquire) >> dev & 1)) return ok;
        std::lock_guard<std::mutex> lock(mu);
        if (kept && (done.load(std::memory_order_relaxed) >> dev & 1)) return ok;
        const R r = f();
        if (kept && r == ok) done.fetch_or(1ull << dev, std::memory_order_release);
        return r;
    }
};

}  // namespace impec
