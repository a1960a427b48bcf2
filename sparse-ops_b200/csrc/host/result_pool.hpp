// result_pool.hpp -- page-locked memory for results that are handed to the caller.
//
// A result copied into a fresh pageable array costs the driver's bounce buffer and a page fault per
// 4 KB (4 MB: 290 us and more); the device writes page-locked memory at link speed (77 us).  Locking
// pages is itself slow, so blocks are kept when a result is released and given to a later one.  The
// pool is bounded: at most kMaxLive results hold a block at a time and kMaxBytes are locked in all; a
// program that keeps more results than that gets ordinary arrays for the others.
#pragma once

#include <cstddef>
#include <mutex>
#include <vector>

#include "spx_b200.h"

namespace spx {

class ResultPool {
public:
    static constexpr size_t kMinBytes = 64 * 1024;      // below, a plain array is as fast
    static constexpr size_t kMaxBytes = size_t(256) << 20;
    static constexpr int kMaxLive = 8;

    struct Block {
        void* ptr;
        size_t bytes;
    };

    static ResultPool& get() {
        static ResultPool* p = new ResultPool();        // never destroyed: results may outlive the module
        return *p;
    }
    // {nullptr, 0} when the caller should use ordinary memory.
    Block acquire(size_t bytes) {
        if (bytes < kMinBytes || bytes > kMaxBytes / 2) return {nullptr, 0};
        const size_t want = (bytes + kMinBytes - 1) / kMinBytes * kMinBytes;
        std::vector<Block> drop;
        Block out{nullptr, 0};
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (live_ >= kMaxLive) return out;
            for (size_t i = 0; i < free_.size(); ++i)
                if (free_[i].bytes >= want && free_[i].bytes <= 2 * want) {
                    out = free_[i];
                    free_.erase(free_.begin() + i);
                    ++live_;
                    return out;
                }
            while (!free_.empty() && total_ + want > kMaxBytes) {       // the oldest make room
                drop.push_back(free_.front());
                total_ -= free_.front().bytes;
                free_.erase(free_.begin());
            }
            if (total_ + want <= kMaxBytes) {
                total_ += want;
                ++live_;
                out.bytes = want;
            }
        }
        for (const Block& b : drop) spx_host_free(b.ptr);
        if (out.bytes && spx_host_alloc(&out.ptr, want) != SPX_OK) {
            std::lock_guard<std::mutex> lk(mu_);
            total_ -= want;
            --live_;
            out = {nullptr, 0};
        }
        return out;
    }
    void release(const Block& b) {
        std::lock_guard<std::mutex> lk(mu_);
        --live_;
        free_.push_back(b);
    }

private:
    std::mutex mu_;
    std::vector<Block> free_;
    size_t total_ = 0;          // bytes locked: handed out and free
    int live_ = 0;
};

}  // namespace spx
