// First touch of pageable host memory that the device is about to copy into.
// Host code only.
#pragma once

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <initializer_list>
#include <thread>
#include <vector>

namespace axs {

// First touch of a pageable destination, ahead of the copies into it. Copies
// into pages that exist run at the link's rate (134 MB in 0.72 ms); into fresh
// ones (a new numpy array) one thread takes the page faults inside the copy,
// 5.6 ms. Up to six threads write one byte per page, chunk by chunk (every byte
// is overwritten by the copy), so that the faults of the next chunks run beside
// the copy of this one. Small destinations are left to the copy, null ones skipped.
class Touch {
  public:
    Touch(std::initializer_list<void *> dst, size_t bytes, size_t chunk_bytes) : bytes_(bytes), chunk_(chunk_bytes) {
        for (void *d : dst)
            if (d) dst_.push_back(d);
        if (bytes * dst_.size() < ((size_t)8 << 20)) return;
        const int n = (int)std::min<unsigned>(6, std::max(1u, std::thread::hardware_concurrency() / 2));
        try {
            done_ = std::vector<std::atomic<int>>((bytes + chunk_ - 1) / chunk_);
            threads_.reserve(n);
            for (int t = 0; t < n; ++t) threads_.emplace_back([this, t, n] { work(t, n); });
        } catch (...) {   // no memory or no thread: the copies take the faults
            join();       // a byte written from here on could land on one that a copy has brought
            done_.clear();
        }
    }
    ~Touch() { join(); }
    Touch(const Touch &) = delete;
    void wait(size_t c) {   // until chunk c's pages exist
        if (done_.empty()) return;
        while (done_[c] < (int)threads_.size()) std::this_thread::yield();
    }

  private:
    void join() {
        stop_ = true;
        for (std::thread &t : threads_) t.join();
        threads_.clear();
    }
    void work(int t, int n) {
        const size_t page = (size_t)std::max(4096l, sysconf(_SC_PAGESIZE));
        for (size_t c = 0; c < done_.size() && !stop_; ++c) {
            const size_t lo = c * chunk_, len = std::min(chunk_, bytes_ - lo), a = lo + len / n * t,
                         b = t == n - 1 ? lo + len : lo + len / n * (t + 1);
            for (void *d : dst_)
                for (size_t o = a; o < b && !stop_; o = (o / page + 1) * page) ((volatile char *)d)[o] = 0;
            ++done_[c];
        }
    }
    std::vector<void *> dst_;
    size_t bytes_, chunk_;
    std::vector<std::atomic<int>> done_;
    std::atomic<bool> stop_{false};
    std::vector<std::thread> threads_;
};

}  // namespace axs
