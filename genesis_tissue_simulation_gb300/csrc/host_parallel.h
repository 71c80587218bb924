// Independent host work over a few threads.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <optional>
#include <thread>
#include <vector>

namespace gbt {

// A few threads that run one loop after another.  run(n, body) calls body(i, worker) for i in [0, n), worker
// below threads(); the calling thread is worker 0.  A thread takes about 20 us to start and 20 us to end in a large
// process, so the first one starts the others while the caller goes on, a loop does not wait for a thread
// that has not begun to work on it, and after dismiss the threads end while the caller goes on (the destructor
// waits for them).  A thread that cannot be started is done without; the first exception of a body is thrown
// by run.
class Team {
public:
    explicit Team(int threads) : size_(std::max(1, std::min((int)std::thread::hardware_concurrency(), threads))) {
        if (size_ == 1) return;
        try {
            pool_.reserve(size_ - 2);
            first_ = std::thread([this]() {
                try {
                    for (int t = 2; t < size_ && !stop_; t++) pool_.emplace_back([this, t]() { work(t); });
                } catch (...) {   // fewer threads
                }
                work(1);
            });
        } catch (...) {   // the caller alone
        }
    }
    ~Team() {
        dismiss();
        if (first_.joinable()) first_.join();   // after it nobody adds to the pool
        for (auto& t : pool_) t.join();
    }
    Team(const Team&) = delete;
    Team& operator=(const Team&) = delete;
    int threads() const { return size_; }
    template <class Body> void run(int n, Body&& body) {
        if (!first_.joinable() || n <= 1 || stop_) {
            for (int i = 0; i < n; i++) body(i, 0);
            return;
        }
        auto loop = [&](int worker) { for (int i; (i = next_++) < n;) body(i, worker); };
        {
            const std::lock_guard<std::mutex> hold(lock_);
            next_ = 0;
            call_ = [](void* f, int worker) { (*(decltype(loop)*)f)(worker); };
            body_ = &loop;
            failed_ = nullptr;
            round_++;
            open_ = true;
        }
        wake_.notify_all();
        guarded(0);
        std::unique_lock<std::mutex> hold(lock_);
        open_ = false;   // nobody joins the loop any more
        done_.wait(hold, [&]() { return working_ == 0; });
        if (failed_) std::rethrow_exception(failed_);
    }
    // After the last loop (a further one is run by the caller alone).
    void dismiss() {
        {
            const std::lock_guard<std::mutex> hold(lock_);
            stop_ = true;
        }
        wake_.notify_all();
    }

private:
    const int size_;
    std::thread first_;
    std::vector<std::thread> pool_;
    std::mutex lock_;
    std::condition_variable wake_, done_;
    std::atomic<int> next_{0};
    std::atomic<bool> stop_{false};
    void (*call_)(void*, int) = nullptr;
    void* body_ = nullptr;
    int working_ = 0;
    unsigned round_ = 0;
    bool open_ = false;
    std::exception_ptr failed_;

    void guarded(int worker) {
        try {
            call_(body_, worker);
        } catch (...) {
            next_ = 1 << 30;   // the others stop at their next index
            const std::lock_guard<std::mutex> hold(lock_);
            if (!failed_) failed_ = std::current_exception();
        }
    }
    void work(int worker) {
        unsigned seen = 0;
        std::unique_lock<std::mutex> hold(lock_);
        for (;;) {
            wake_.wait(hold, [&]() { return stop_ || (open_ && round_ != seen); });
            if (stop_) return;
            seen = round_;
            working_++;
            hold.unlock();
            guarded(worker);
            hold.lock();
            if (--working_ == 0) done_.notify_one();
        }
    }
};

// A team kept by `place` beyond its use, so that the wait for its threads' ends falls on the next use or the
// owner's close; it is dismissed with the scope at the latest.
struct BriefTeam {
    Team& team;
    BriefTeam(std::optional<Team>& place, int threads) : team(place.emplace(threads)) {}
    ~BriefTeam() { team.dismiss(); }
};

// One loop on up to `threads` threads.
template <class Body> void parallelFor(int n, int threads, Body&& body) {
    Team team(std::min(threads, n));
    team.run(n, [&](int i, int) { body(i); });
}

}  // namespace gbt
