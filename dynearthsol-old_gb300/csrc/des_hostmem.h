// Whether a kernel may read or write ordinary host memory in place.
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>
#include <vector>

namespace des {

// Whether every page of the range is in memory (true below 1 MB without a
// look).  A page that nobody has touched yet is brought in by the GPU's access
// one fault at a time, 5 to 10 times slower than by a copy through the driver:
// a frame of 2.4M elements into fresh arrays 84 ms against 13.5, uploading
// untouched zeros 205 against 23, the closure's outputs of 4M samples 42
// against 7.3; on touched pages it is in place that is faster (frame 2.5
// against 2.9, upload 3.85 against 4.8).  Unmapped ranges are not in memory.
inline bool pages_present(const void *p, size_t bytes)
{
    if (bytes < (size_t)1 << 20) return true;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = reinterpret_cast<uintptr_t>(p) & ~(page - 1),
                    e = reinterpret_cast<uintptr_t>(p) + bytes;
    std::vector<unsigned char> in((e - a + page - 1) / page);
    if (mincore(reinterpret_cast<void *>(a), e - a, in.data())) return false;
    for (unsigned char c : in)
        if (!(c & 1)) return false;
    return true;
}

// Whether the first and the last page of the range may be read (written): an
// array that the program may not write makes the GPU's store a fault of the
// whole context, where the driver's copy can refuse.  (The pages are brought in
// as the access would do.  Kernels before Linux 5.14 say no to everything.)
inline bool pages_allow(const void *p, size_t bytes, bool write)
{
#ifndef MADV_POPULATE_READ
    enum { MADV_POPULATE_READ = 22, MADV_POPULATE_WRITE = 23 };
#endif
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = reinterpret_cast<uintptr_t>(p) & ~(page - 1),
                    z = (reinterpret_cast<uintptr_t>(p) + bytes - 1) & ~(page - 1);
    const int advice = write ? MADV_POPULATE_WRITE : MADV_POPULATE_READ;
    return !madvise(reinterpret_cast<void *>(a), page, advice) &&
           (z == a || !madvise(reinterpret_cast<void *>(z), page, advice));
}

}  // namespace des
