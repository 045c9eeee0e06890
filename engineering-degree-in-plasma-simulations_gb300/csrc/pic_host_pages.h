// First touch of the pages of a caller's host array (host code only).
#pragma once
#include <sys/mman.h>
#include <unistd.h>
#include <algorithm>
#include <cstddef>
#include <thread>

namespace pic {

// Makes the pages of a caller's array that is to be filled from the device present and writable, and leaves its
// values as they are, so that a call that fails later has not touched them.  A copy into an untouched
// allocation faults page by page from the copy's side, which took between 0.08 and 6.6 ms for 8 MB from
// call to call, against 0.05 ms into pages that are there.  The faults zero the pages at the speed of one core, 32
// GB/s, so large arrays share them among up to kTouchThreads threads, each with kTouchBytes at least (a thread
// costs about as much as the faults of 1 MB).  madvise does it without a write: 134 MB of fresh pages take 3.6
// ms with one thread, 1.6 with four, 2.6 with eight, which wait for one another's lock; 403 MB 12.1, 4.5, 7.8.
// (Writing zeros instead takes 1.1 and 2.8 ms with eight threads, atomic additions of zero 6.1 and 14.3.)  Where
// the system does not know the advice, or not for this mapping, the pages come with the copy.
#ifdef MADV_POPULATE_WRITE
constexpr int kPopulateWrite = MADV_POPULATE_WRITE;
#else
constexpr int kPopulateWrite = 23;  // Linux 5.14
#endif
constexpr size_t kTouchBytes = 8u << 20;
constexpr int kTouchThreads = 4;
inline void touch_pages(void* out, size_t bytes) {
    static const size_t page = (size_t)std::max(4096l, sysconf(_SC_PAGESIZE));
    if (!bytes) return;
    // whole pages, the first and the last also where the array has a part of them
    const size_t first = reinterpret_cast<size_t>(out) / page, pages = (reinterpret_cast<size_t>(out) + bytes - 1) / page + 1 - first;
    auto touch = [first](size_t from, size_t to) {
        if (from < to) madvise(reinterpret_cast<void*>((first + from) * page), (to - from) * page, kPopulateWrite);
    };
    const size_t n = std::max<size_t>(1, std::min<size_t>(kTouchThreads, bytes / kTouchBytes)), share = (pages + n - 1) / n;
    std::thread helper[kTouchThreads];
    size_t started = 1;
    for (; started < n; started++) try {
            helper[started] = std::thread(touch, std::min(pages, started * share), std::min(pages, (started + 1) * share));
        } catch (...) {
            break;  // no thread or no memory for one: the caller's own takes the rest
        }
    touch(0, std::min(pages, share));
    if (started < n) touch(std::min(pages, started * share), pages);
    for (size_t t = 1; t < started; t++) helper[t].join();
}

}  // namespace pic
