// Independent host work over a few threads.
#pragma once
#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

namespace gbt {

// Runs body(i) for i in [0, n) on up to 16 host threads.
template <class Body> void parallelFor(int n, Body&& body) {
    const int threads = std::max(1, std::min({(int)std::thread::hardware_concurrency(), 16, n}));
    std::atomic<int> next{0};
    auto run = [&]() { for (int i; (i = next++) < n;) body(i); };
    std::vector<std::thread> pool;
    for (int t = 1; t < threads; t++) pool.emplace_back(run);
    run();
    for (auto& t : pool) t.join();
}

}  // namespace gbt
