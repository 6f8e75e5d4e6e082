// Host check of pb::PerDevice (prism_b200/csrc/common.h) against a fake current device: the
// value is found on every device's own first use and kept there, from several threads too.
#include "../../prism_b200/csrc/common.h"

#include <cstdio>
#include <thread>

namespace {
thread_local int g_device = 0;  // the fake current device (the runtime keeps one per thread, too)
}
extern "C" {
cudaError_t cudaGetDevice(int* d) {
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

int main() {
    pb::PerDevice value;
    std::atomic<int> found[200] = {};
    auto get = [&] { return value.get([&] { return ++found[g_device], 100 + g_device; }); };
    for (int round = 0; round < 3; ++round)
        for (int d : {0, 1, 5, 63}) {
            g_device = d;
            if (get() != 100 + d || found[d] != 1) return std::fprintf(stderr, "device %d\n", d), 1;
        }
    g_device = 150;  // beyond the table: found each time
    if (get() != 250 || get() != 250 || found[150] != 2) return std::fprintf(stderr, "large ordinal\n"), 1;
    std::vector<std::thread> threads;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int k = 0; k < 1000; ++k) {
                g_device = 10 + (t + k) % 20;
                if (get() != 100 + g_device) ++wrong;
            }
        });
    for (auto& t : threads) t.join();
    return wrong ? 1 : 0;
}
