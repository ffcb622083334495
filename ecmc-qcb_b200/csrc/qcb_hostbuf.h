// qcb_hostbuf.h -- host buffers that are used again (the server's copies of the requests' links).  Plain C++.
#pragma once
#include <stdlib.h>

#include <mutex>
#include <vector>

namespace qcb {

struct HostBuf {
    void* p = nullptr;
    size_t cap = 0;
};

class HostBufs {
  public:
    // At most `limit` bytes wait for another use.
    explicit HostBufs(size_t limit) : limit_(limit) {}
    HostBufs(const HostBufs&) = delete;
    HostBufs& operator=(const HostBufs&) = delete;
    ~HostBufs() {
        for (HostBuf& b : free_) free(b.p);
    }

    // A buffer of at least n bytes (p = NULL: out of memory): the smallest free one that does, unless it is
    // more than four times as large, or a new one.
    HostBuf take(size_t n) {
        HostBuf b;
        {
            std::lock_guard<std::mutex> lk(mu_);
            size_t best = free_.size();
            for (size_t i = 0; i < free_.size(); i++) {
                const size_t cap = free_[i].cap;
                if (cap >= n && cap / 4 <= n && (best == free_.size() || cap < free_[best].cap)) best = i;
            }
            if (best < free_.size()) {
                b = free_[best];
                free_.erase(free_.begin() + (long)best);
                bytes_ -= b.cap;
                return b;
            }
        }
        b.p = malloc(n);
        b.cap = n;
        return b;
    }

    // Back for another use.  One of more than the limit is freed and the others stay; else the oldest leave
    // where they would hold more than that together.
    void give(HostBuf b) {
        if (b.cap > limit_ || !keep(b)) {
            free(b.p);
            return;
        }
        for (;;) {
            HostBuf old;
            {
                std::lock_guard<std::mutex> lk(mu_);
                if (bytes_ <= limit_) return;
                old = free_.front();
                free_.erase(free_.begin());
                bytes_ -= old.cap;
            }
            free(old.p);
        }
    }

  private:
    bool keep(HostBuf b) {
        std::lock_guard<std::mutex> lk(mu_);
        try {
            free_.push_back(b);
        } catch (...) {
            return false;
        }
        bytes_ += b.cap;
        return true;
    }
    const size_t limit_;
    std::mutex mu_;
    std::vector<HostBuf> free_;
    size_t bytes_ = 0;
};

}  // namespace qcb
