// Page faults of a large host result, taken while the GPU works.
//
// A result array fresh from the allocator has no pages yet, and a device-to-host
// copy into it faults them in one by one: 44 MB take 2.4 ms on the Grace host
// (64 KiB pages), 0.25 ms into pages that the GPU has seen before, 0.93 into new
// ones.  Helper threads ask the kernel for the pages (MADV_POPULATE_WRITE, which
// leaves the contents alone; 44 MB in 1.0 ms with one thread, 0.68 with two, 0.6
// with four; touching the pages from user space 2.2 ms with any number) as soon
// as the call knows the array, part by part, and the copy waits for them, whole
// or part by part.  A kernel without the call, or memory that it does not apply
// to, only loses the saving.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <system_error>
#include <thread>

namespace rectv {

class ResultPages {
  public:
    static constexpr size_t kMinBytes = size_t(4) << 20;  // smaller arrays: about the cost of the threads
    static constexpr int kThreads = 4, kParts = 8;

    ResultPages(void *p, size_t bytes) : base_((uintptr_t)p), bytes_(bytes), parts_(bytes < kMinBytes ? 1 : kParts) {
        if (parts_ == 1) return;
        for (int i = 0; i < kThreads; ++i) {
            try {
                t_[i] = std::thread([this, i] {
                    for (int k = i; k < kParts; k += kThreads) {
                        populate(k);
                        std::lock_guard<std::mutex> lk(mu_);
                        done_ |= 1u << k;
                        cv_.notify_all();
                    }
                });
            } catch (const std::system_error &) {  // no thread to be had: the copy takes the faults
                std::lock_guard<std::mutex> lk(mu_);
                for (int k = i; k < kParts; k += kThreads) done_ |= 1u << k;
            }
        }
    }
    ResultPages(const ResultPages &) = delete;
    ResultPages &operator=(const ResultPages &) = delete;
    ~ResultPages() {
        for (std::thread &t : t_)
            if (t.joinable()) t.join();
    }
    // the array in parts: bytes [begin(k), begin(k + 1)) of part k
    int parts() const { return parts_; }
    size_t begin(int k) const { return k >= parts_ ? bytes_ : bytes_ / parts_ / 4096 * 4096 * k; }
    void wait(int k) {
        if (parts_ == 1) return;
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return (done_ >> k) & 1u; });
    }
    void wait() {
        for (int k = 0; k < parts_; ++k) wait(k);
    }

  private:
    void populate(int k) const {
        constexpr int populate_write = 23;  // MADV_POPULATE_WRITE (absent from older headers)
        const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
        // the pages that begin in the part and lie in the array
        const uintptr_t a = (base_ + begin(k) + page - 1) / page * page;
        const uintptr_t b = std::min((base_ + begin(k + 1) + page - 1) / page * page, (base_ + bytes_) / page * page);
        if (a < b) (void)madvise((void *)a, b - a, populate_write);
    }
    uintptr_t base_;
    size_t bytes_;
    int parts_;
    unsigned done_ = 0;
    std::mutex mu_;
    std::condition_variable cv_;
    std::thread t_[kThreads];
};

}  // namespace rectv
