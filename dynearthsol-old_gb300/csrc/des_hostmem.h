// Makes ordinary host memory ready for a kernel to read or write in place.
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

#ifndef MADV_POPULATE_READ
#define MADV_POPULATE_READ 22
#define MADV_POPULATE_WRITE 23
#endif

namespace des {

// whether every page from a to e (page boundaries) is in memory
inline bool pages_present(uintptr_t a, uintptr_t e)
{
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    unsigned char in[4096];
    for (uintptr_t at = a; at < e;) {
        const size_t n = std::min<size_t>(sizeof in, (e - at) / page);
        if (mincore(reinterpret_cast<void *>(at), n * page, in)) return false;
        for (size_t k = 0; k < n; ++k)
            if (!(in[k] & 1)) return false;
        at += n * page;
    }
    return true;
}

// the pages from a to e brought in as the access would do, a thread for every
// 16 MB up to four; false where one may not be accessed
inline bool populate(uintptr_t a, uintptr_t e, int advice)
{
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    const int parts = (int)std::min<size_t>(4, std::max<size_t>(1, (e - a) >> 24));
    const size_t each = ((e - a) / parts + page - 1) / page * page;
    std::atomic<bool> ok{true};
    auto part = [&](uintptr_t from) {
        if (from < e && madvise(reinterpret_cast<void *>(from), std::min(each, (size_t)(e - from)), advice)) ok = false;
    };
    std::vector<std::thread> others;
    int k = 1;
    try {
        others.reserve(parts);
        for (; k < parts; ++k) others.emplace_back(part, a + k * each);
    } catch (const std::exception &) {       // (no thread to be had: the rest here)
    }
    for (; k < parts; ++k) part(a + k * each);
    part(a);
    for (std::thread &t : others) t.join();
    return ok;
}

// Whether a kernel may read (write) the range in place.  A page that nobody has
// touched yet is brought in here: by the GPU's own access it takes a fault of
// its own, 5 to 10 times as long (a frame of 2.4M elements into fresh arrays 84
// ms against 7.3; 13.4 by a copy through the driver, up to 130 where the copy
// engine is cold).  And an access that the program may not make itself is
// left for the driver's copy to refuse: the GPU's would end the context.  Pages
// that are there cost a look (6 us for 128 MB) and a try of the first and the
// last.  (Before Linux 5.14: no.)
inline bool pages_ready(const void *p, size_t bytes, bool write)
{
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = reinterpret_cast<uintptr_t>(p) & ~(page - 1),
                    e = (reinterpret_cast<uintptr_t>(p) + bytes + page - 1) & ~(page - 1);
    const int advice = write ? MADV_POPULATE_WRITE : MADV_POPULATE_READ;
    if (e - a <= 2 * page || !pages_present(a, e)) return populate(a, e, advice);
    return populate(a, a + page, advice) && populate(e - page, e, advice);
}

}  // namespace des
