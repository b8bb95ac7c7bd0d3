// CopyPool: every part runs once; a second copy gets threads while the first one holds its own; where no thread can be started
// the caller copies alone; a forked child copies alone and ends; the threads end with the last user.  Prints "ok" or the line
// that failed.
#include "copy_pool.hpp"

#include <sys/resource.h>
#include <sys/wait.h>

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <filesystem>
#include <fstream>
#include <set>
#include <string>

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::fflush(stdout); _exit(1); } } while (0)

static bool wait_for(const std::function<bool()>& what) {
    for (int i = 0; i < 5000; ++i) {
        if (what()) return true;
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
    }
    return false;
}
static int threads_of_process() {
    int n = 0;
    for (auto it = std::filesystem::directory_iterator("/proc/self/task"); it != std::filesystem::directory_iterator(); ++it) ++n;
    return n;
}
static bool all_parts_once(fdk::CopyPool& pool) {
    std::atomic<int> covered[24] = {};   // 24 = what every number of parts up to 8 divides, or nearly
    pool.run([&](int part, int parts) {
        for (int i = 24 * part / parts; i < 24 * (part + 1) / parts; ++i) ++covered[i];
    });
    for (auto& c : covered) if (c != 1) return false;
    return true;
}
template <typename F>
static bool child_ends_well(F&& f) {
    const pid_t pid = fork();
    if (pid == 0) {
        alarm(20);
        std::exit(f() ? 0 : 1);
    }
    int status = 0;
    waitpid(pid, &status, 0);
    return WIFEXITED(status) && WEXITSTATUS(status) == 0;
}

int main() {
    // no memory for a thread's stack: before this process has threads of its own
    CHECK(child_ends_well([] {
        size_t pages = 0;
        std::ifstream("/proc/self/statm") >> pages;
        const rlim_t now = (rlim_t)pages * (rlim_t)sysconf(_SC_PAGESIZE) + (1 << 20);
        const rlimit lim{now, now};
        if (setrlimit(RLIMIT_AS, &lim) != 0) return false;
        fdk::CopyPool pool(7);
        return all_parts_once(pool) && all_parts_once(pool);
    }));
    {
        fdk::CopyPool alone(0);
        CHECK(all_parts_once(alone));
    }
    {
        fdk::CopyPool pool(14);
        for (int i = 0; i < 200; ++i) CHECK(all_parts_once(pool));
        // the first copy's parts wait until the second copy is done
        std::atomic<int> holding{0};
        std::atomic<bool> go{false};
        std::thread first([&] { pool.run([&](int, int) { ++holding; CHECK(wait_for([&] { return go.load(); })); }); });
        CHECK(wait_for([&] { return holding.load() == fdk::CopyPool::PARTS; }));
        std::atomic<int> inside{0};
        pool.run([&](int, int) { ++inside; CHECK(wait_for([&] { return inside.load() >= 4; })); });   // four threads at least
        go = true;
        first.join();
        std::thread callers[4];
        for (auto& t : callers) t = std::thread([&] { for (int i = 0; i < 200; ++i) CHECK(all_parts_once(pool)); });
        for (auto& t : callers) t.join();
        CHECK(child_ends_well([&] { return all_parts_once(pool); }));
    }
    CHECK(threads_of_process() == 1);
    {
        auto a = fdk::CopyPool::shared(), b = fdk::CopyPool::shared();
        CHECK(a == b && all_parts_once(*a));
        CHECK(child_ends_well([&] { const bool ok = all_parts_once(*a); a.reset(); b.reset(); return ok; }));
    }
    CHECK(wait_for([] { return threads_of_process() == 1; }));
    std::printf("ok\n");
}
