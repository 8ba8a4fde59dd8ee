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
// the calling thread and returns when every call is done. Workers start on first use and
// stop with the owning context.
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
            active_ = workers_.size();
            ++gen_;
        }
        cv_.notify_all();
        drain();
        std::unique_lock<std::mutex> lk(mu_);
        done_cv_.wait(lk, [&] { return active_ == 0; });
        fn_ = nullptr;
    }

private:
    void drain() {
        for (uint64_t i; (i = next_.fetch_add(1)) < n_;) (*fn_)(i);
    }
    void start() {
        if (started_) return;
        started_ = true;
        const unsigned hw = std::thread::hardware_concurrency();
        const unsigned nt = hw > 1 ? std::min(7u, hw - 1) : 0u;
        for (unsigned t = 0; t < nt; ++t) workers_.emplace_back([this] { loop(); });
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            std::unique_lock<std::mutex> lk(mu_);
            cv_.wait(lk, [&] { return quit_ || gen_ != seen; });
            if (quit_) return;
            seen = gen_;
            lk.unlock();
            drain();
            lk.lock();
            if (--active_ == 0) done_cv_.notify_one();
        }
    }
    std::vector<std::thread> workers_;
    std::mutex mu_;
    std::condition_variable cv_, done_cv_;
    const std::function<void(uint64_t)>* fn_ = nullptr;
    uint64_t n_ = 0, gen_ = 0;
    std::atomic<uint64_t> next_{0};
    size_t active_ = 0;
    bool quit_ = false, started_ = false;
};

}  // namespace ndtgb
