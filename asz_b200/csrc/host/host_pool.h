// Worker threads kept for a context's host-side parallel loops.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace asz::host {

// run(n, f) calls f(0..n-1) on the workers and the calling thread, and returns when all calls have
// returned. It does not wait for workers that found nothing left to do: waking all of them costs
// more than a small loop.
class HostPool {
public:
    explicit HostPool(unsigned workers) {
        for (unsigned i = 0; i < workers; i++) th_.emplace_back([this] { loop(); });
    }
    ~HostPool() {
        {
            std::lock_guard<std::mutex> g(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto &t : th_) t.join();
    }
    void run(uint64_t n, const std::function<void(uint64_t)> &f) {
        if (n == 0) return;
        if (n == 1 || th_.empty()) {
            for (uint64_t j = 0; j < n; j++) f(j);
            return;
        }
        auto job = std::make_shared<Job>(f, n);
        {
            std::lock_guard<std::mutex> g(mu_);
            job_ = job;
            ++gen_;
        }
        cv_.notify_all();
        job->work();
        std::unique_lock<std::mutex> l(job->mu);
        job->done_cv.wait(l, [&] { return job->done == n; });
    }

private:
    // A worker that comes late holds its job, and finds nothing left in it.
    struct Job {
        Job(const std::function<void(uint64_t)> &fn, uint64_t count) : f(fn), n(count) {}
        void work() {
            uint64_t mine = 0;
            for (uint64_t j; (j = next.fetch_add(1)) < n; mine++) f(j);  // f outlives its last call
            if (!mine) return;
            std::lock_guard<std::mutex> g(mu);
            done += mine;
            if (done == n) done_cv.notify_all();
        }
        const std::function<void(uint64_t)> &f;
        const uint64_t n;
        std::atomic<uint64_t> next{0};
        std::mutex mu;
        std::condition_variable done_cv;
        uint64_t done = 0;
    };
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            std::shared_ptr<Job> job;
            {
                std::unique_lock<std::mutex> l(mu_);
                cv_.wait(l, [&] { return stop_ || gen_ != seen; });
                if (stop_) return;
                seen = gen_;
                job = job_;
            }
            job->work();
        }
    }
    std::vector<std::thread> th_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::shared_ptr<Job> job_;
    uint64_t gen_ = 0;
    bool stop_ = false;
};

}  // namespace asz::host
