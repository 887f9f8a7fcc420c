// PerDevice against a stand-in for the runtime's current device: each device makes its own value once, a failure
// is not kept, and threads agree.
#include "kernels/per_device.hpp"

#include <cstdio>
#include <thread>
#include <vector>

static thread_local int g_device = 0;
cudaError_t cudaGetDevice(int* dev) {
    *dev = g_device;
    return cudaSuccess;
}

int main() {
    tdg::PerDevice c;
    int made[3] = {}, bad = 0;
    auto value = [&](int dev) {
        g_device = dev;
        return c.get([&] { return ++made[dev], 10 + dev; });
    };
    for (int round = 0; round < 2; ++round)
        for (int dev = 0; dev < 3; ++dev) bad += value(dev) != 10 + dev;
    for (int dev = 0; dev < 3; ++dev) bad += made[dev] != 1;
    tdg::PerDevice d;
    g_device = 1;
    bad += d.get([] { return 0; }) != 0;
    bad += d.get([] { return 5; }) != 5;
    bad += d.get([] { return 6; }) != 5;
    g_device = 1000;  // beyond the cache: made every time
    bad += d.get([] { return 7; }) != 7 || d.get([] { return 8; }) != 8;
    tdg::PerDevice e;
    std::vector<std::thread> ts;
    std::vector<int> seen(16);
    for (int i = 0; i < 16; ++i)
        ts.emplace_back([&, i] {
            g_device = i % 4;
            for (int k = 0; k < 1000; ++k) seen[i] = e.get([&] { return 1 + i % 4; });
        });
    for (auto& t : ts) t.join();
    for (int i = 0; i < 16; ++i) bad += seen[i] != 1 + i % 4;
    std::printf("%d\n", bad);
    return 0;
}
