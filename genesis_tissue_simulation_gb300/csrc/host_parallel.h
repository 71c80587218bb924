// Independent host work over a few threads.
#pragma once
#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace gbt {

// Runs body(i, workspace) for i in [0, n) on up to `threads` threads, each with a workspace of its own.  A
// thread that cannot be started is done without; the first exception of a body is thrown here.
template <class Workspace, class Body> void parallelFor(int n, int threads, Workspace&& workspace, Body&& body) {
    threads = std::max(1, std::min({(int)std::thread::hardware_concurrency(), threads, n}));
    std::atomic<int> next{0};
    std::mutex lock;
    std::exception_ptr failed;
    auto run = [&]() {
        try {
            auto own = workspace();
            for (int i; (i = next++) < n;) body(i, own);
        } catch (...) {
            const std::lock_guard<std::mutex> hold(lock);
            if (!failed) failed = std::current_exception();
            next = n;
        }
    };
    std::vector<std::thread> pool;
    try {
        for (int t = 1; t < threads; t++) pool.emplace_back(run);
    } catch (...) {   // fewer threads
    }
    run();
    for (auto& t : pool) t.join();
    if (failed) std::rethrow_exception(failed);
}
template <class Body> void parallelFor(int n, Body&& body) {
    parallelFor(n, 16, []() { return 0; }, [&](int i, int&) { body(i); });
}

}  // namespace gbt
