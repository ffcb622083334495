// qcb_hostbuf.h -- host buffers that are used again, and wait for the end of a copy before that.
//
// A server takes a buffer for each request's links, fills it, starts a copy from it to the device and gives
// it back with the event that follows the copy.  Another thread may fill a buffer the moment it takes it,
// so one whose copy has not ended is never handed out.  Plain C++: Event is a cudaEvent_t in the server.
#pragma once
#include <stdlib.h>

#include <mutex>
#include <vector>

namespace qcb {

struct HostBuf {
    void* p = nullptr;
    size_t cap = 0;
};

template <class Event>
class HostBufs {
  public:
    // At most `limit` bytes wait for another use.
    explicit HostBufs(size_t limit) : limit_(limit) {}
    HostBufs(const HostBufs&) = delete;
    HostBufs& operator=(const HostBufs&) = delete;
    ~HostBufs() {
        for (HostBuf& b : free_) free(b.p);
        for (Copy& c : copies_) free(c.b.p);
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

    // Back once the copy that `done` follows has ended.  False without memory to note it: b stays the caller's.
    bool give_after(HostBuf b, Event done) {
        std::lock_guard<std::mutex> lk(mu_);
        try {
            copies_.push_back(Copy{b, done});
        } catch (...) {
            return false;
        }
        return true;
    }
    // Gives back the buffers whose event `ended` finds complete, and hands each such event to `release`.
    template <class Ended, class Release>
    void reclaim(Ended ended, Release release) {
        for (;;) {
            Copy c;
            {
                std::lock_guard<std::mutex> lk(mu_);
                size_t i = 0;
                while (i < copies_.size() && !ended(copies_[i].done)) i++;
                if (i == copies_.size()) return;
                c = copies_[i];
                copies_.erase(copies_.begin() + (long)i);
            }
            release(c.done);
            give(c.b);
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
    struct Copy {
        HostBuf b;
        Event done;
    };
    const size_t limit_;
    std::mutex mu_;
    std::vector<HostBuf> free_;
    size_t bytes_ = 0;
    std::vector<Copy> copies_;
};

}  // namespace qcb
