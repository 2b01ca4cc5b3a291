// First touch of pageable host memory that the device is about to copy into.
// Host code only.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <thread>
#include <vector>

namespace axs {

// First touch of a pageable destination, ahead of the copies into it. Copies
// into pages that exist run at the link's rate (134 MB in 0.72 ms); into fresh
// ones (a new numpy array) one thread takes the page faults inside the copy,
// 5.6 ms. Up to six threads write one byte into each page that is not there yet, chunk
// by chunk (every byte is overwritten by the copy), so that the faults of the
// next chunks run beside the copy of this one. Where fewer than 8 MB are
// missing, the arrays of a program that keeps them, no thread is started:
// starting six costs 0.2 ms, as much as copying 40 MB. Null destinations are skipped.
class Touch {
  public:
    static constexpr size_t kLeast = (size_t)8 << 20;
    Touch(std::initializer_list<void *> dst, size_t bytes, size_t chunk_bytes) : bytes_(bytes), chunk_(chunk_bytes) {
        if (bytes * dst.size() < kLeast) return;
        try {
            size_t missing = 0;
            for (void *d : dst)
                if (d && bytes) missing += add((char *)d);
            if (missing * page_ < kLeast) return;
            const int n = (int)std::min<unsigned>(6, std::max(1u, std::thread::hardware_concurrency() / 2));
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
    struct Dst {
        char *p;
        std::vector<unsigned char> there;   // bit 0: the page exists; the first page is p's
    };
    // Takes a destination in; returns the number of its pages that do not exist yet.
    size_t add(char *p) {
        const size_t head = (uintptr_t)p % page_;
        Dst d{p, std::vector<unsigned char>((head + bytes_ + page_ - 1) / page_)};
        if (mincore(p - head, head + bytes_, d.there.data()) != 0) return 0;   // not wholly mapped: the copy's to report
        size_t missing = 0;
        for (unsigned char c : d.there) missing += !(c & 1);
        if (missing) dst_.push_back(std::move(d));
        return missing;
    }
    void work(int t, int n) {
        for (size_t c = 0; c < done_.size() && !stop_; ++c) {
            const size_t lo = c * chunk_, len = std::min(chunk_, bytes_ - lo), a = lo + len / n * t,
                         b = t == n - 1 ? lo + len : lo + len / n * (t + 1);
            for (const Dst &d : dst_) {
                const size_t head = (uintptr_t)d.p % page_;
                for (size_t o = a; o < b && !stop_;) {
                    const size_t i = (head + o) / page_;
                    if (!(d.there[i] & 1)) ((volatile char *)d.p)[o] = 0;
                    o = (i + 1) * page_ - head;
                }
            }
            ++done_[c];
        }
    }
    const size_t page_ = (size_t)std::max(4096l, sysconf(_SC_PAGESIZE));
    std::vector<Dst> dst_;
    size_t bytes_, chunk_;
    std::vector<std::atomic<int>> done_;
    std::atomic<bool> stop_{false};
    std::vector<std::thread> threads_;
};

}  // namespace axs
