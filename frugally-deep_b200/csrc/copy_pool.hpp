// Host threads that copy memory together: what moves a caller's pageable or scattered samples into page-locked staging memory
// (one thread copies about 10 GB/s, the bus takes five times that).  Several callers (one per device) may have a copy under
// way; up to 7 threads are started for each of them, no more than half of the cores in all, and every thread takes parts
// from the copies in turn.  A caller takes parts of its own copy as well, so that it gets done whatever the threads do, also
// where none could be started or (in a forked child) none exists.
#pragma once

#include <unistd.h>

#include <algorithm>
#include <condition_variable>
#include <deque>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace fdk {

class CopyPool {
public:
    static constexpr int PARTS = 8;
    // The pool of the process; its threads end with the last of its users.
    static std::shared_ptr<CopyPool> shared() {
        static std::mutex mu;
        static std::weak_ptr<CopyPool> known;
        std::lock_guard<std::mutex> lk(mu);
        std::shared_ptr<CopyPool> p = known.lock();
        if (!p) known = p = std::make_shared<CopyPool>(std::max(0, (int)std::thread::hardware_concurrency() / 2 - 1));
        return p;
    }
    explicit CopyPool(int most_threads) : s_(std::make_unique<State>()) { s_->most = most_threads; }
    CopyPool(const CopyPool&) = delete;
    CopyPool& operator=(const CopyPool&) = delete;
    ~CopyPool() {
        if (getpid() != pid_) {
            s_.release();   // a forked child: the threads are the parent's; nothing here can be joined or waited out
            return;
        }
        {
            std::lock_guard<std::mutex> lk(s_->mu);
            s_->stop = true;
        }
        s_->wake.notify_all();
        for (auto& t : s_->workers) t.join();
    }
    // job(part, PARTS) for every part, side by side; returns when all are done.  The job must not throw.
    void run(const std::function<void(int, int)>& job) {
        if (getpid() != pid_) {
            job(0, 1);
            return;
        }
        State& s = *s_;
        Copy own{&job};
        std::unique_lock<std::mutex> lk(s.mu);
        s.copies.push_back(&own);
        ++s.active;
        while ((int)s.workers.size() < std::min(s.most, (PARTS - 1) * s.active)) {
            try {
                s.workers.emplace_back([&s] { s.work(); });
            } catch (const std::exception&) {
                s.most = (int)s.workers.size();   // no more threads to be had
            }
        }
        s.wake.notify_all();
        while (own.next < PARTS) s.take(lk, own);
        s.done.wait(lk, [&] { return own.done == PARTS; });
        --s.active;
    }

private:
    struct Copy {
        const std::function<void(int, int)>* job;
        int next = 0, done = 0;
    };
    struct State {
        int most = 0;
        int active = 0;
        bool stop = false;
        std::mutex mu;
        std::condition_variable wake, done;
        std::deque<Copy*> copies;   // those with parts left
        std::vector<std::thread> workers;
        // One part of a copy that has parts left; mu is held on entry and on return.
        void take(std::unique_lock<std::mutex>& lk, Copy& c) {
            const int part = c.next++;
            copies.erase(std::find(copies.begin(), copies.end(), &c));
            if (c.next < PARTS) copies.push_back(&c);   // behind the others
            lk.unlock();
            (*c.job)(part, PARTS);
            lk.lock();
            if (++c.done == PARTS) done.notify_all();
        }
        void work() {
            std::unique_lock<std::mutex> lk(mu);
            for (;;) {
                wake.wait(lk, [&] { return stop || !copies.empty(); });
                if (stop) return;
                take(lk, *copies.front());
            }
        }
    };
    const pid_t pid_ = getpid();
    std::unique_ptr<State> s_;
};

}  // namespace fdk
