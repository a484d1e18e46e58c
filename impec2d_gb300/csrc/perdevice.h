// Host-side state that exists once per device of a process (no CUDA types: also compiled alone by the tests).
#pragma once
#include <mutex>

namespace impec {

// Something each device needs once, such as a kernel's shared-memory limit: do_once(dev, ok, f) calls f until it has
// returned ok for that device.  Devices beyond the 64 that are remembered call f every time, which does
// no harm.  Safe with several threads; f runs under the lock.
class OncePerDevice {
    std::mutex mu;
    unsigned long long done = 0;

public:
    template <class R, class F>
    R do_once(int dev, R ok, F&& f) {
        std::lock_guard<std::mutex> lock(mu);
        const bool kept = dev >= 0 && dev < 64;
        if (kept && (done >> dev & 1)) return ok;
        const R r = f();
        if (kept && r == ok) done |= 1ull << dev;
        return r;
    }
};

}  // namespace impec
