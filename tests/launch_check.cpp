// PerDevice (fcb_launch.hpp): every device is set up, once, with its own numbers; a failed
// setup runs again; threads that launch at the same time read complete numbers.
#include <cstdio>
#include <thread>
#include <vector>

#include "../forestclaw_b200/csrc/fcb_launch.hpp"

int main() {
    int wrong = 0;
    fcb::PerDevice<2> kept;
    int setups[4] = {};
    auto ask = [&](int dev, bool fail) {
        int out[2] = {-1, -1};
        const int e = kept.get(dev, out, [&](int* n) {
            ++setups[dev];
            n[0] = 10 * dev;
            n[1] = 10 * dev + 1;
            return fail ? 7 : 0;
        });
        if (e != (fail ? 7 : 0)) ++wrong;
        if (!fail && (out[0] != 10 * dev || out[1] != 10 * dev + 1)) ++wrong;
    };
    ask(1, true);
    for (int k = 0; k < 3; ++k)
        for (int dev = 0; dev < 4; ++dev) ask(dev, false);
    for (int dev = 0; dev < 4; ++dev) wrong += setups[dev] != (dev == 1 ? 2 : 1);

    int none[2], calls = 0;
    for (int k = 0; k < 2; ++k) kept.get(fcb::PerDevice<2>::kDevices, none, [&](int* n) { ++calls; n[0] = n[1] = 0; return 0; });
    wrong += calls != 2;

    static fcb::PerDevice<2> shared;
    std::vector<std::thread> ts;
    int bad[8] = {};
    for (int t = 0; t < 8; ++t)
        ts.emplace_back([&, t] {
            for (int k = 0; k < 20000; ++k) {
                const int dev = k % 64;
                int out[2] = {-1, -1};
                const int e = shared.get(dev, out, [&](int* n) { n[0] = dev + 5; n[1] = dev + 6; return 0; });
                bad[t] += e != 0 || out[0] != dev + 5 || out[1] != dev + 6;
            }
        });
    for (auto& t : ts) t.join();
    for (int b : bad) wrong += b;
    std::printf("%d wrong\n", wrong);
    return wrong != 0;
}
