// First touch of the pages of a caller's host array (host code only).
#pragma once
#include <unistd.h>
#include <algorithm>
#include <cstddef>
#include <thread>

namespace pic {

// Writes to every page of a caller's array that is to be filled from the device: a copy into an untouched
// allocation faults page by page from the copy's side, which took between 0.08 and 6.6 ms for 8 MB from
// call to call, against 0.05 ms into touched pages and about 0.25 ms for the faults on the host.  (A
// read before the write would map the shared zero page first and then replace it, which costs a
// translation shootdown per page: measured 20 us each.)  The faults zero the pages at the speed of one
// core, 32 GB/s, so large arrays share them among up to kTouchThreads threads, each with kTouchBytes at least
// (a thread costs about as much as the faults of 1 MB): 134 MB of potential 5.2 -> 2.3 ms a read,
// 403 MB of field 15.4 -> 5.4.
constexpr size_t kTouchBytes = 8u << 20;
constexpr int kTouchThreads = 8;
inline void touch_pages(void* out, size_t bytes) {
    static const size_t page = (size_t)std::max(4096l, sysconf(_SC_PAGESIZE));
    auto touch = [out, bytes](size_t from, size_t to) {
        volatile char* p = static_cast<volatile char*>(out);
        for (size_t x = from; x < to; x += page) p[x] = 0;
        if (to == bytes && bytes) p[bytes - 1] = 0;
    };
    const int n = (int)std::min<size_t>(kTouchThreads, bytes / kTouchBytes);
    const size_t share = n > 1 ? (bytes / n + page - 1) / page * page : bytes;  // whole pages a thread
    std::thread helper[kTouchThreads];
    int started = 1;
    for (; started < n; started++) try {
            helper[started] = std::thread(touch, std::min(bytes, started * share), std::min(bytes, (started + 1) * share));
        } catch (...) {
            break;  // no thread or no memory for one: the caller's own takes the rest
        }
    touch(0, std::min(bytes, share));
    if (started < n) touch(std::min(bytes, started * share), bytes);
    for (int t = 1; t < started; t++) helper[t].join();
}

}  // namespace pic
