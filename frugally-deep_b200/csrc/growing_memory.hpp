// Device memory that grows with what is asked of it and never moves: a larger request is served from a further block, and
// the blocks before it stay until the owner lets all of them go, so that an address that a recorded launch holds remains
// valid.  Sizes are powers of two, so that all blocks together are less than twice the largest.
#pragma once

#include <chrono>
#include <cstdint>
#include <vector>

namespace fdk {

class GrowingMemory {
public:
    static constexpr int64_t SMALLEST = 1 << 16;   // floats
    // Memory for `floats` values or null.  alloc(floats): the memory, or null where there is none; not called unless
    // may_allocate, and for a second after a failure only for less than what failed (a failing allocation takes up to a
    // millisecond, and the requests of a model's layers come by the dozen).
    template <typename Alloc>
    float* get(int64_t floats, bool may_allocate, Alloc&& alloc, std::chrono::steady_clock::time_point now = std::chrono::steady_clock::now()) {
        if (floats <= size_) return blocks_.back();
        if (!may_allocate || (refused_ > 0 && floats >= refused_ && now - refused_at_ < std::chrono::seconds(1))) return nullptr;
        int64_t size = SMALLEST;
        while (size < floats) size *= 2;
        float* p = alloc(size);
        if (!p && size > floats) p = alloc(size = floats);
        if (!p) {
            refused_ = floats;
            refused_at_ = now;
            return nullptr;
        }
        refused_ = 0;
        size_ = size;
        blocks_.push_back(p);
        return p;
    }
    template <typename Free>
    void release(Free&& free) {
        for (float* p : blocks_) free(p);
        blocks_.clear();
        size_ = 0;
    }

private:
    std::vector<float*> blocks_;
    int64_t size_ = 0;      // of the last block
    int64_t refused_ = 0;   // the last request that found no memory
    std::chrono::steady_clock::time_point refused_at_;
};

}  // namespace fdk
