// GrowingMemory: addresses stay, growth by powers of two, no allocation where it is not allowed, a refusal is not repeated
// within a second but for less, and what there was before it still serves.  Prints "ok" or the line that failed.
#include "growing_memory.hpp"

#include <cstdio>
#include <deque>

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    using fdk::GrowingMemory;
    std::deque<float> heap;   // one float per block: addresses are all that counts
    int64_t left = 1 << 20, asked = 0, last = 0;
    auto alloc = [&](int64_t n) -> float* {
        ++asked;
        if (n > left) return nullptr;
        left -= n;
        last = n;
        heap.push_back(0.f);
        return &heap.back();
    };
    const auto t0 = std::chrono::steady_clock::now();
    GrowingMemory m;
    CHECK(m.get(1, false, alloc, t0) == nullptr && asked == 0);
    float* a = m.get(1, true, alloc, t0);
    CHECK(a && last == GrowingMemory::SMALLEST);
    CHECK(m.get(GrowingMemory::SMALLEST, false, alloc, t0) == a && asked == 1);
    CHECK(m.get(GrowingMemory::SMALLEST + 1, false, alloc, t0) == nullptr);
    float* b = m.get(GrowingMemory::SMALLEST + 1, true, alloc, t0);
    CHECK(b && b != a && last == 2 * GrowingMemory::SMALLEST);
    CHECK(m.get(7, true, alloc, t0) == b);
    asked = 0;
    CHECK(m.get(left + 1, true, alloc, t0) == nullptr && asked >= 1);          // more than there is
    asked = 0;
    CHECK(m.get(left + 2, true, alloc, t0 + std::chrono::milliseconds(999)) == nullptr && asked == 0);
    CHECK(m.get(5, true, alloc, t0) == b);
    left = 5 * GrowingMemory::SMALLEST - 1;
    float* d = m.get(left, true, alloc, t0);                                    // less than what failed; its power of two is not to be had
    CHECK(d && last == 5 * GrowingMemory::SMALLEST - 1);
    left = 1 << 30;
    CHECK(m.get(1 << 20, true, alloc, t0 + std::chrono::seconds(2)) != nullptr);
    int released = 0;
    m.release([&](float*) { ++released; });
    CHECK(released == 4 && m.get(1, false, alloc, t0) == nullptr);
    std::printf("ok\n");
}
