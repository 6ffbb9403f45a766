// Large blocks of device memory that buffers gave back, kept for the next solve on the device.
//
// A solve frees and allocates gigabytes.  From the device's pool a block freed on one stream and taken
// on another (several handles in turn) is often not reusable yet, and the pool maps new memory instead
// (measured: 30-70 ms of a 3x10 solve or a 32-parameter sweep, once 1.1 s).  Kept blocks belong to the
// device, not to a handle: the first solve of a new handle takes what idle handles gave back, and a
// refused allocation gets back everything that is kept, whoever gave it.
//
// A block is taken by the handle that gave it at once (both uses are ordered on its stream), by another
// only when the event recorded as it was given has passed, so no solve waits for another.  At most
// max_held bytes are kept per device; a handle's blocks go back to the pool when it closes or gets an
// HBM budget.  Plain C++ over Api (event and free calls), so that the accounting runs without a device.
#pragma once
#include <cstddef>
#include <mutex>
#include <vector>

namespace momed {

template <class Api>
class KeptBlocks {
public:
    using Stream = typename Api::Stream;
    using Event = typename Api::Event;
    static constexpr size_t kMinBlock = size_t(1) << 20;

    explicit KeptBlocks(size_t max_held = size_t(16) << 30) : max_held_(max_held) {}

    // A block of at least `bytes`, at most a quarter larger; null: none.  (Larger ones given to the pool
    // to carve the allocation from are missed by the next request of their size: 25 -> 47 ms for a mixed
    // 3x9 solve on handles in turn.)
    void* take(size_t bytes, const void* owner, size_t& got) {
        std::lock_guard<std::mutex> lk(mu_);
        size_t best = blocks_.size();
        for (size_t i = 0; i < blocks_.size(); ++i)
            if (blocks_[i].bytes >= bytes && blocks_[i].bytes <= bytes + bytes / 4 &&
                (best == blocks_.size() || blocks_[i].bytes < blocks_[best].bytes) && ready(blocks_[i], owner))
                best = i;
        if (best == blocks_.size()) return nullptr;
        const Block b = remove(best);
        got = b.bytes;
        return b.p;
    }

    // False: not kept, the caller frees the block.
    bool put(void* p, size_t bytes, const void* owner, Stream st) noexcept {
        if (bytes < kMinBlock || bytes > max_held_) return false;
        try {
            std::lock_guard<std::mutex> lk(mu_);
            for (size_t i = 0; held_ + bytes > max_held_;) {            // oldest first
                while (i < blocks_.size() && !ready(blocks_[i], owner)) ++i;
                if (i == blocks_.size()) return false;
                Api::free(remove(i).p, st);
            }
            blocks_.reserve(blocks_.size() + 1);
            idle_.reserve(blocks_.size() + 1 + idle_.size());
            Event e;
            if (!idle_.empty()) {
                e = idle_.back();
                idle_.pop_back();
            } else if (!Api::create(e)) {
                return false;
            }
            if (!Api::record(e, st)) {
                idle_.push_back(e);
                return false;
            }
            blocks_.push_back({p, bytes, owner, e});
            held_ += bytes;
            return true;
        } catch (...) {
            return false;
        }
    }

    // The owner's blocks back to the pool; st: the stream its buffers are ordered on.
    void drop(const void* owner, Stream st) noexcept {
        std::lock_guard<std::mutex> lk(mu_);
        for (size_t i = blocks_.size(); i-- > 0;)
            if (blocks_[i].owner == owner) Api::free(remove(i).p, st);
    }

    // Everything back to the pool, ordered on st behind the givers' work; false: nothing was kept.
    bool reclaim(Stream st) noexcept {
        std::lock_guard<std::mutex> lk(mu_);
        if (blocks_.empty()) return false;
        for (size_t i = blocks_.size(); i-- > 0;) {
            Api::wait(st, blocks_[i].given);
            Api::free(remove(i).p, st);
        }
        return true;
    }

    size_t held() {
        std::lock_guard<std::mutex> lk(mu_);
        return held_;
    }

private:
    struct Block {
        void* p;
        size_t bytes;
        const void* owner;
        Event given;
    };
    bool ready(const Block& b, const void* owner) { return b.owner == owner || Api::passed(b.given); }
    Block remove(size_t i) {
        const Block b = blocks_[i];
        blocks_.erase(blocks_.begin() + i);
        held_ -= b.bytes;
        idle_.push_back(b.given);                        // within the capacity that put reserved
        return b;
    }
    std::mutex mu_;
    std::vector<Block> blocks_;                          // oldest first
    std::vector<Event> idle_;                            // events of blocks that left
    size_t held_ = 0, max_held_;
};

}  // namespace momed
