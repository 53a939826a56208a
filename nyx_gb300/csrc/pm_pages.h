// Host pages of a buffer that a device-to-host copy is about to fill.
//
// On a host whose page tables the GPU shares, a copy into pages the process has not touched
// yet takes a GPU page fault for each (measured 1.4 to 25 GB/s against 190 GB/s into pages that
// are there).  touch_pages has the host fault them in before the copy and writes nothing:
// until the copy runs the buffer holds what it held, whatever the call's outcome.  Missing
// pages come in by the kernel (MADV_POPULATE_WRITE), which refuses an address the process
// cannot write (a read-only mapping, device memory) where a store would end the process.
// Which are missing says mincore (0.35 us and 3.5 us for 50 MB of 64 KB pages).  Pages that are there are
// read: without it a read-back of 470 MB into them took 20 to 60 ms instead of 6 about every
// half second, as if their entries had been closed in between.
//
// Measured on fresh pages: 8 MB 161 us (186 by a store to each page), 20 MB 221 (198), 50 MB 500
// (456), 400 MB 3440 (3890); three threads up to 128 MB, as four wait for one another in the
// kernel (50 MB 84 GB/s against 103; 400 MB 113 against 92), in steps of 1 MB (in one step per
// thread 64 GB/s).  Pages that are there: 8 MB 0.9 us, 50 MB 40, 400 MB 87 (0.2, 35, 49).
// (A page that was read before its first write counts as there: the copy faults it.)
#pragma once

#include <cstddef>
#include <cstdint>
#include <thread>

#include <sys/mman.h>
#include <unistd.h>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace nyxpm {

constexpr size_t kPageStep = (size_t)1 << 20;            // bytes brought in per system call
constexpr size_t kPageLook = (size_t)16 << 20;           // bytes asked about per system call
constexpr size_t kPageMin = 4096;
constexpr size_t kTouchThreadsFrom = (size_t)16 << 20;   // bytes worth threads
constexpr size_t kTouchThreeTo = (size_t)128 << 20;      // missing bytes better by three than by four
constexpr size_t kReadThreadsFrom = (size_t)128 << 20;   // bytes worth threads to read only

// the missing pages of [at, end), whole pages; touch: fault them in and read the others
inline size_t missing_pages(uintptr_t at, uintptr_t end, size_t page, bool touch)
{
    unsigned char there[kPageLook / kPageMin];
    const size_t step = kPageStep / page;
    size_t missing = 0, look = kPageLook;
    while (at < end) {
        const size_t len = end - at < look ? end - at : look, pages = len / page;
        if (mincore(reinterpret_cast<void*>(at), len, there) != 0) {
            if (look == kPageStep) return missing;   // not mapped
            look = kPageStep;
            continue;
        }
        for (size_t i0 = 0; i0 < pages; i0 += step) {
            const size_t i1 = i0 + step < pages ? i0 + step : pages;
            size_t first = i1, last = 0;
            for (size_t i = i0; i < i1; ++i) {
                if (there[i] & 1) {
                    if (touch) (void)*reinterpret_cast<volatile char*>(at + i * page);
                    continue;
                }
                ++missing;
                if (first == i1) first = i;
                last = i;
            }
            if (touch && first < i1)
                madvise(reinterpret_cast<void*>(at + first * page), (last + 1 - first) * page, MADV_POPULATE_WRITE);
        }
        at += len;
    }
    return missing;
}

inline void fill_pages(uintptr_t at, uintptr_t end, size_t page) { missing_pages(at, end, page, true); }

inline void read_pages(uintptr_t at, uintptr_t end, size_t page)
{
    for (; at < end; at += page) (void)*reinterpret_cast<volatile char*>(at);
}

// work on the whole pages of [at, end) in up to four threads, the caller's among them
inline void pages_by_threads(void (*work)(uintptr_t, uintptr_t, size_t), uintptr_t at, uintptr_t end, size_t page,
                             int threads)
{
    std::thread t[3];
    const size_t part = (end - at) / threads & ~(kPageStep - 1);
    try {
        for (int k = 0; k + 1 < threads; ++k) {
            t[k] = std::thread(work, at, at + part, page);
            at += part;
        }
    } catch (...) {   // no more threads, or no memory for one: the rest here
    }
    work(at, end, page);
    for (std::thread& x : t)
        if (x.joinable()) x.join();
}

// there: no page is missing, as of pinned memory
inline void touch_pages(void* p, size_t bytes, bool there = false)
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    if (!p || !bytes || page < kPageMin || page > kPageStep) return;
    const uintptr_t at = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)(page - 1);
    const uintptr_t end = (reinterpret_cast<uintptr_t>(p) + bytes + page - 1) & ~(uintptr_t)(page - 1);
    if (there) return pages_by_threads(read_pages, at, end, page, end - at < kReadThreadsFrom ? 1 : 4);
    int threads = 1;
    if (end - at >= kTouchThreadsFrom) {
        const size_t missing = missing_pages(at, end, page, false) * page;
        threads = missing >= kTouchThreadsFrom && missing < kTouchThreeTo ? 3 : 4;
    }
    pages_by_threads(fill_pages, at, end, page, threads);
}

}  // namespace nyxpm
