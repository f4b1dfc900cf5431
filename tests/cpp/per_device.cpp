// PerDevice: a value of its own for each device, made once, whichever thread asks.
#include <cstdio>
#include <thread>
#include <vector>

#include "per_device.hpp"

int main() {
    rkdg::PerDevice<int> kept;
    int made[2] = {0, 0};
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; ++i)
        threads.emplace_back([&, i] {
            for (int k = 0; k < 1000; ++k)
                kept.use(i % 2, [&](int& v) {
                    if (v == 0) v = 10 + i % 2, ++made[i % 2];
                    return v;
                });
        });
    for (auto& t : threads) t.join();
    std::printf("%d %d %d %d\n", kept.use(0, [](int& v) { return v; }), kept.use(1, [](int& v) { return v; }), made[0], made[1]);
    return 0;
}
