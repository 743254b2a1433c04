// Pages of a buffer in pageable memory, made ahead of a copy into it.  Plain host code: the thread that makes them makes no
// CUDA call, so it needs no device of its own, and whoever starts it decides what memory it may touch.
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <exception>
#include <thread>

namespace b200 {

// In fresh memory the faults are a good part of a copy to the host (neighbour lists in arrays that no call had before, whole
// call, ms, without and with: 20,000 x 32, K = 32 3.3, 1.9; 100,003 x 96, K = 32 11.8, 9.6; 200,000 x 16, K = 20 14.4, 8.5).
// Small buffers and those that several threads will fill are left alone (two lists of 150 MB, pages made ahead of the
// threads: 28 -> 50 ms).
constexpr size_t kPopulateMin = (size_t)2 << 20, kPopulateEnd = (size_t)24 << 20;
inline bool worth_populating(size_t bytes) { return bytes >= kPopulateMin && bytes < kPopulateEnd; }

// Gives the buffer's whole pages memory, and leaves its contents as they are.  It looks at `stop` between pieces, so that
// whoever is ready to copy does not wait for the rest.
inline void populate_pages(void *p, size_t bytes, const std::atomic<bool> &stop)
{
#ifdef MADV_POPULATE_WRITE
    if (!p || !worth_populating(bytes)) return;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), lo = ((uintptr_t)p + page - 1) / page * page, hi = ((uintptr_t)p + bytes) / page * page;
    constexpr uintptr_t piece = (uintptr_t)1 << 20;
    // a failure (an old kernel, a mapping of another kind) leaves the faults to the copy
    for (uintptr_t at = lo; at < hi && !stop.load(std::memory_order_relaxed); at += piece)
        if (madvise(reinterpret_cast<void *>(at), std::min(piece, hi - at), MADV_POPULATE_WRITE) != 0) return;
#else
    (void)p;
    (void)bytes;
    (void)stop;
#endif
}

// The pages that a buffer lacks.  All are looked at (1 us a megabyte at most): arrays from an allocator that recycles memory have
// some of theirs, in any place.
inline size_t pages_missing(const void *p, size_t bytes)
{
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), lo = ((uintptr_t)p + page - 1) / page * page, hi = ((uintptr_t)p + bytes) / page * page;
    size_t missing = 0;
    unsigned char in[1024];
    for (uintptr_t at = lo; p && at < hi;) {
        const size_t n = std::min<size_t>(sizeof(in), (hi - at) / page);
        if (mincore(reinterpret_cast<void *>(at), n * page, in) != 0) return 0;   // no ordinary memory
        for (size_t k = 0; k < n; k++) missing += !(in[k] & 1);
        at += n * page;
    }
    return missing;
}
// A buffer that an earlier call has filled needs no thread: starting one and waiting for it takes 25 us, what the faults of as many
// pages take (9,000 x 20, K = 60 into arrays that have theirs 759 us with a thread, 719 without; and a thread in each call
// changes what the C library gives back: 8,353 x 106, K = 99 1.35 -> 2.3 ms).
constexpr size_t kPagesWorthAThread = 18;

// A thread that populates up to two buffers of one size until it is told that the copy is due.
class PagesAhead {
public:
    PagesAhead() = default;
    PagesAhead(const PagesAhead &) = delete;
    PagesAhead &operator=(const PagesAhead &) = delete;
    ~PagesAhead() { end(); }
    void start(void *a, void *b, size_t bytes)   // null: none
    {
        if (thread_.joinable() || !worth_populating(bytes) || pages_missing(a, bytes) + pages_missing(b, bytes) < kPagesWorthAThread) return;
        try {
            thread_ = std::thread([this, a, b, bytes] {
                populate_pages(a, bytes, stop_);
                populate_pages(b, bytes, stop_);
            });
        } catch (const std::exception &) {   // no thread to be had: the copy finds the pages itself
        }
    }
    bool started() const { return thread_.joinable(); }
    void end()
    {
        stop_ = true;
        if (thread_.joinable()) thread_.join();
        stop_ = false;
    }

private:
    std::thread thread_;
    std::atomic<bool> stop_{false};
};

}  // namespace b200
