// host_pool.h — host threads for staging copies (internal).
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace ndtgb {

// A few host threads for staging copies: run(n, f) calls f(0 .. n-1) across the workers and
// the calling thread and returns when every call is done. A worker that has not yet woken by
// then finds nothing to enter: waiting for all seven to report cost a call of a few short copies
// about 45 us. Workers start on first use (or by start()) and stop with the owning context.
class HostPool {
public:
    ~HostPool() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            quit_ = true;
        }
        cv_.notify_all();
        for (auto& w : workers_) w.join();
    }
    void run(uint64_t n, const std::function<void(uint64_t)>& f) {
        if (n == 0) return;
        start();
        if (workers_.empty() || n == 1) {
            for (uint64_t i = 0; i < n; ++i) f(i);
            return;
        }
        {
            std::lock_guard<std::mutex> lk(mu_);
            fn_ = &f;
            n_ = n;
            next_.store(0);
            ++gen_;
        }
        cv_.notify_all();
        drain(f, n);
        // every item is taken: none may enter any more, those inside finish theirs
        std::unique_lock<std::mutex> lk(mu_);
        fn_ = nullptr;
        done_cv_.wait(lk, [&] { return inside_ == 0; });
    }
    void start() {
        if (started_) return;
        started_ = true;
        const unsigned hw = std::thread::hardware_concurrency();
        const unsigned nt = hw > 1 ? std::min(7u, hw - 1) : 0u;
        for (unsigned t = 0; t < nt; ++t) workers_.emplace_back([this] { loop(); });
    }

private:
    void drain(const std::function<void(uint64_t)>& f, uint64_t n) {
        for (uint64_t i; (i = next_.fetch_add(1)) < n;) f(i);
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            std::unique_lock<std::mutex> lk(mu_);
            cv_.wait(lk, [&] { return quit_ || (fn_ && gen_ != seen); });
            if (quit_) return;
            seen = gen_;
            const std::function<void(uint64_t)>& f = *fn_;
            const uint64_t n = n_;
            ++inside_;
            lk.unlock();
            drain(f, n);
            lk.lock();
            if (--inside_ == 0) done_cv_.notify_one();
        }
    }
    std::vector<std::thread> workers_;
    std::mutex mu_;
    std::condition_variable cv_, done_cv_;
    const std::function<void(uint64_t)>* fn_ = nullptr;
    uint64_t n_ = 0, gen_ = 0;
    std::atomic<uint64_t> next_{0};
    size_t inside_ = 0;  // workers at the current items
    bool quit_ = false, started_ = false;
};

}  // namespace ndtgb
