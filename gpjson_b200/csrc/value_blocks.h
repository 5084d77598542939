// Host memory of gathered values (gpj_query_values).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <utility>
#include <vector>

namespace gpj {

// Page-locked memory (copied to at full speed, no page faults) up to kMost in
// all, free blocks kept for later values of the process until its last context
// is destroyed.  Beyond it pageable memory.  `Pages` page-locks and frees:
// void* Pages::lock(size_t) (null: cannot), void Pages::unlock(void*).
template <class Pages>
class ValueBlocks {
  public:
    static constexpr size_t kMost = size_t(64) << 20;

    uint8_t* take(size_t size, size_t* cap, bool* pinned) {
        const size_t exact = (size + 0xFFFF) & ~size_t(0xFFFF);
        size_t want = exact;
        *pinned = true;
        {
            std::lock_guard<std::mutex> g(mu_);
            // A block of about the size; a new one beside the free ones
            // (larger than asked where sizes vary: the next may need it);
            // any block; a new one in place of the free ones.  So that a few
            // values do not hold the block of many, nor values of two sizes
            // in turn have their memory page-locked each time.
            if (uint8_t* p = pick(size, 2 * size + (size_t(1) << 20), cap)) return p;
            if (!free_.empty()) want = (size + size / 4 + 0xFFFF) & ~size_t(0xFFFF);
            if (total_ + want > kMost) want = exact;
            if (total_ + want > kMost) {
                if (uint8_t* p = pick(size, kMost, cap)) return p;
                drop_free();
            }
            if (total_ + want > kMost)
                want = 0;
            else
                total_ += want;
        }
        if (want) {
            if (void* p = Pages::lock(want)) {
                *cap = want;
                return static_cast<uint8_t*>(p);
            }
            std::lock_guard<std::mutex> g(mu_);
            total_ -= want;
        }
        *pinned = false;
        *cap = size;
        void* p = std::malloc(size);
        if (p) std::memset(p, 0, size);  // a copy that faults in its own pages is slower
        return static_cast<uint8_t*>(p);
    }

    void give(uint8_t* p, size_t cap, bool pinned) {
        if (!p) return;
        if (!pinned) {
            std::free(p);
            return;
        }
        std::lock_guard<std::mutex> g(mu_);
        try {
            if (contexts_ > 0) {
                free_.emplace_back(p, cap);
                return;
            }
        } catch (const std::exception&) {
            // no room to note it
        }
        total_ -= cap;
        Pages::unlock(p);
    }

    void context_created() {
        std::lock_guard<std::mutex> g(mu_);
        ++contexts_;
    }
    void context_destroyed() {
        std::lock_guard<std::mutex> g(mu_);
        if (--contexts_ == 0) drop_free();
    }

  private:
    // The smallest free block of [size, largest] bytes, or null.
    uint8_t* pick(size_t size, size_t largest, size_t* cap) {
        size_t best = free_.size();
        for (size_t i = 0; i < free_.size(); i++)
            if (free_[i].second >= size && free_[i].second <= largest &&
                (best == free_.size() || free_[i].second < free_[best].second))
                best = i;
        if (best == free_.size()) return nullptr;
        const auto b = free_[best];
        free_.erase(free_.begin() + best);
        *cap = b.second;
        return b.first;
    }
    void drop_free() {
        for (auto& b : free_) {
            total_ -= b.second;
            Pages::unlock(b.first);
        }
        free_.clear();
    }

    std::mutex mu_;
    std::vector<std::pair<uint8_t*, size_t>> free_;
    size_t total_ = 0;  // page-locked bytes, in use or free
    int contexts_ = 0;
};

}  // namespace gpj
