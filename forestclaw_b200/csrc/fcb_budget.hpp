// A bound on memory that many owners keep for their next use.
#pragma once
#include <atomic>
#include <cstddef>

namespace fcb {

// One owner's share, of at most `own` bytes, of a total of at most `cap` that all owners
// add to (any threads).
class KeptBytes {
  public:
    KeptBytes(std::atomic<size_t>& total, size_t own, size_t cap) : total_(total), own_(own), cap_(cap) {}
    KeptBytes(const KeptBytes&) = delete;
    KeptBytes& operator=(const KeptBytes&) = delete;
    ~KeptBytes() { clear(); }
    // the owner keeps n bytes more, or may not
    bool add(size_t n) {
        if (n > own_ - mine_) return false;
        size_t t = total_.load(std::memory_order_relaxed);
        do {
            if (n > cap_ || t > cap_ - n) return false;
        } while (!total_.compare_exchange_weak(t, t + n, std::memory_order_relaxed));
        mine_ += n;
        return true;
    }
    void clear() {
        total_.fetch_sub(mine_, std::memory_order_relaxed);
        mine_ = 0;
    }

  private:
    std::atomic<size_t>& total_;
    const size_t own_, cap_;
    size_t mine_ = 0;
};

}  // namespace fcb
