// pinned_cache.h -- free page-locked blocks kept between the handles that use
// them (memory.cu).  Plain C++: which blocks are handed out, kept and dropped.
//
// The blocks belong to the context of the device they were allocated for.  A
// process may have handles on several devices, whose contexts live side by
// side; a block is taken for gone only when its own device's context is another
// one now (cudaDeviceReset took it, and its address may be in use again, so it
// is forgotten, not freed).
#pragma once

#include <stddef.h>

#include <vector>

namespace dyg {

class PinnedCache {
public:
    explicit PinnedCache(size_t limit) : limit_(limit) {}

    // A kept block of exactly `bytes` from this device's present context, or null.
    void *take(int dev, unsigned long long ctx, size_t bytes) {
        for (size_t i = blocks_.size(); i-- > 0;) {
            const Block b = blocks_[i];
            if (b.dev != dev || b.ctx != ctx || b.bytes != bytes) continue;
            drop(i);
            return b.p;
        }
        return nullptr;
    }

    // Keeps the block if there is room for it; false: the caller frees it.
    bool keep(int dev, unsigned long long ctx, void *p, size_t bytes) {
        for (size_t i = blocks_.size(); i-- > 0;)
            if (blocks_[i].dev == dev && blocks_[i].ctx != ctx) drop(i);
        if (total_ + bytes > limit_) return false;
        blocks_.push_back(Block{p, bytes, ctx, dev});
        total_ += bytes;
        return true;
    }

    size_t total() const { return total_; }

private:
    struct Block {
        void *p;
        size_t bytes;
        unsigned long long ctx;
        int dev;
    };
    void drop(size_t i) {
        total_ -= blocks_[i].bytes;
        blocks_[i] = blocks_.back();
        blocks_.pop_back();
    }
    std::vector<Block> blocks_;
    size_t total_ = 0, limit_;
};

}  // namespace dyg
