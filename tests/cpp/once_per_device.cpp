// Host-side check of OncePerDevice: one call per device, again after a failure, every time beyond the devices
// that are remembered, one call when many threads ask at once.  Prints "ok" or the first thing that is wrong.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "perdevice.h"

static void expect(bool ok, const char* what) {
    if (ok) return;
    std::printf("%s\n", what);
    std::exit(1);
}

int main() {
    impec::OncePerDevice once;
    int calls[70] = {0};
    auto set = [&](int dev, int result) {
        return once.do_once(dev, 0, [&] { ++calls[dev]; return result; });
    };
    expect(set(0, 0) == 0 && set(0, 0) == 0 && calls[0] == 1, "device 0: not exactly one call");
    expect(set(1, 0) == 0 && calls[1] == 1, "device 1 was not told after device 0");
    expect(set(2, 7) == 7 && calls[2] == 1, "a failure is not reported");
    expect(set(2, 0) == 0 && calls[2] == 2, "no second try after a failure");
    expect(set(2, 0) == 0 && calls[2] == 2, "a third call after success");
    expect(set(63, 0) == 0 && set(63, 0) == 0 && calls[63] == 1, "device 63: not exactly one call");
    expect(set(64, 0) == 0 && set(64, 0) == 0 && calls[64] == 2, "device 64: not a call each time");
    std::atomic<int> n{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 16; ++t)
        ts.emplace_back([&] {
            for (int k = 0; k < 1000; ++k) once.do_once(5, 0, [&] { ++n; return 0; });
        });
    for (auto& t : ts) t.join();
    expect(n == 1, "several calls from several threads");
    std::puts("ok");
}
