// Set-up per device (csrc/per_device.h): once for every device, also from several threads, and again after a failure.
#include "per_device.h"

#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

static int failures = 0;
static void expect(bool ok, const char *what) {
    if (ok) return;
    std::printf("FAILED: %s\n", what);
    ++failures;
}

int main() {
    enn_b200::PerDeviceInit init;
    int calls[3] = {0, 0, 0};
    auto run = [&](int device, int result) { return init.run(device, [&] { return ++calls[device], result; }); };
    expect(run(0, 0) == 0 && run(0, 0) == 0 && calls[0] == 1, "once for a device");
    expect(run(1, 0) == 0 && calls[1] == 1, "a second device gets its own set-up");
    expect(run(2, 7) == 7 && run(2, 0) == 0 && calls[2] == 2, "a failure is returned and not remembered");
    expect(run(2, 9) == 0 && calls[2] == 2, "done after the success");

    enn_b200::PerDeviceInit shared;
    std::atomic<int> count{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] { shared.run(t % 4, [&] { return ++count, 0; }); });
    for (auto &t : threads) t.join();
    expect(count == 4, "once per device from eight threads");
    return failures ? 1 : 0;
}
