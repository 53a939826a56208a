// Host pages of a buffer that a device-to-host copy is about to fill.
//
// On a host whose page tables the GPU shares, a copy into pages the process has not touched
// yet takes a GPU page fault for each (measured 1.4 to 25 GB/s against 190 GB/s into pages that
// are there).  touch_pages has the host fault them in before the copy and writes nothing:
// until the copy runs the buffer holds what it held, whatever the call's outcome.  Missing
// pages come in by the kernel (MADV_POPULATE_WRITE), which refuses an address the process
// cannot write (a read-only mapping, device memory) where a store would end the process.
// Which are missing says mincore (3.5 us for 50 MB of 64 KB pages).  Pages that are there are
// read: without it a read-back of 470 MB into them took 20 to 60 ms instead of 6 about every
// half second, as if their entries had been closed in between.
//
// Measured on fresh pages, GB/s: one thread 48 (a store to each page 42); 16 MB by three threads
// 79 and 50 MB 103 (four threads 72 and 84: they wait for one another in the kernel); 400 MB by
// four 113, by three 92.  In steps of 1 MB: in one step per thread 64 GB/s for 50 MB by four.
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

constexpr size_t kPageStep = (size_t)1 << 20;            // bytes per system call
constexpr size_t kPageMin = 4096;
constexpr size_t kTouchThreadsFrom = (size_t)16 << 20;   // bytes worth threads
constexpr size_t kTouchThreeTo = (size_t)128 << 20;      // missing bytes better by three than by four

// the missing pages of [at, end), whole pages; touch: fault them in and read the others
inline size_t missing_pages(uintptr_t at, uintptr_t end, size_t page, bool touch)
{
    unsigned char there[kPageStep / kPageMin];
    size_t missing = 0;
    while (at < end) {
        const size_t len = end - at < kPageStep ? end - at : kPageStep, pages = len / page;
        if (mincore(reinterpret_cast<void*>(at), len, there) != 0) return missing;   // not mapped
        size_t first = pages, last = 0;
        for (size_t i = 0; i < pages; ++i) {
            if (there[i] & 1) {
                if (touch) (void)*reinterpret_cast<volatile char*>(at + i * page);
                continue;
            }
            ++missing;
            if (first == pages) first = i;
            last = i;
        }
        if (touch && first < pages)
            madvise(reinterpret_cast<void*>(at + first * page), (last + 1 - first) * page, MADV_POPULATE_WRITE);
        at += len;
    }
    return missing;
}

inline void touch_pages(void* p, size_t bytes)
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    if (!p || !bytes || page < kPageMin || page > kPageStep) return;
    uintptr_t at = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)(page - 1);
    const uintptr_t end = (reinterpret_cast<uintptr_t>(p) + bytes + page - 1) & ~(uintptr_t)(page - 1);
    constexpr int kMost = 4;
    std::thread t[kMost - 1];
    if (end - at >= kTouchThreadsFrom) {
        const size_t missing = missing_pages(at, end, page, false) * page;
        const int threads = missing >= kTouchThreadsFrom && missing < kTouchThreeTo ? 3 : kMost;
        const size_t part = (end - at) / threads & ~(kPageStep - 1);
        try {
            for (int k = 0; k + 1 < threads; ++k) {
                t[k] = std::thread(missing_pages, at, at + part, page, true);
                at += part;
            }
        } catch (...) {   // no more threads, or no memory for one: the rest here
        }
    }
    missing_pages(at, end, page, true);
    for (std::thread& x : t)
        if (x.joinable()) x.join();
}

}  // namespace nyxpm
