// A few host threads that copy memory together: what moves a caller's pageable or scattered samples into page-locked staging
// memory (one thread copies about 10 GB/s, the bus takes five times that).  One job at a time; a caller that finds the pool
// busy copies by itself.  Started on first use, at most 7 threads, joined when the process ends.
#pragma once

#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace fdk {

class CopyPool {
public:
    static CopyPool& instance() {
        static CopyPool pool;
        return pool;
    }
    // job(part, parts) for every part in 0 .. parts - 1, in parallel; returns when all are done.  The jobs must not throw.
    void run(const std::function<void(int, int)>& job) {
        std::unique_lock<std::mutex> use(use_, std::try_to_lock);
        if (!use.owns_lock() || workers_.empty()) {
            job(0, 1);
            return;
        }
        const int parts = (int)workers_.size() + 1;
        {
            std::lock_guard<std::mutex> lk(mu_);
            job_ = &job;
            parts_ = parts;
            left_ = parts - 1;
            ++round_;
        }
        wake_.notify_all();
        job(parts - 1, parts);
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [&] { return left_ == 0; });
        job_ = nullptr;
    }

private:
    CopyPool() {
        const int cores = (int)std::thread::hardware_concurrency();
        const int n = std::min(7, std::max(0, cores / 2 - 1));
        for (int i = 0; i < n; ++i) workers_.emplace_back([this, i] { work(i); });
    }
    ~CopyPool() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        wake_.notify_all();
        for (auto& t : workers_) t.join();
    }
    void work(int part) {
        uint64_t seen = 0;
        for (;;) {
            const std::function<void(int, int)>* job;
            int parts;
            {
                std::unique_lock<std::mutex> lk(mu_);
                wake_.wait(lk, [&] { return stop_ || round_ != seen; });
                if (stop_) return;
                seen = round_;
                job = job_;
                parts = parts_;
            }
            (*job)(part, parts);
            {
                std::lock_guard<std::mutex> lk(mu_);
                if (--left_ == 0) done_.notify_one();
            }
        }
    }
    std::mutex use_, mu_;
    std::condition_variable wake_, done_;
    std::vector<std::thread> workers_;
    const std::function<void(int, int)>* job_ = nullptr;
    int parts_ = 0, left_ = 0;
    uint64_t round_ = 0;
    bool stop_ = false;
};

}  // namespace fdk
