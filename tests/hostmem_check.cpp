// Host check of csrc/des_hostmem.h on untouched, touched, partly touched,
// released, protected and unmapped ranges: what pages_ready allows, that the
// pages are there afterwards, and that no byte changes.  exit 1 on a mismatch.
#include "des_hostmem.h"

#include <cstdio>
#include <cstring>

int main()
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = (size_t)34 << 20;
    int bad = 0;
    auto fail = [&](const char *what) { printf("%s\n", what), ++bad; };
    auto map = [&] { return static_cast<char *>(mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0)); };
    auto present = [&](const char *p, size_t bytes) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~(page - 1);
        return des::pages_present(a, (reinterpret_cast<uintptr_t>(p) + bytes + page - 1) & ~(page - 1));
    };
    // untouched ranges of one byte to two threads' worth, from a page's start and its middle
    for (size_t bytes : {(size_t)1, page, 2 * page + 1, ((size_t)33 << 20) + 5})
        for (size_t from : {(size_t)0, (size_t)24}) {
            char *p = map();
            if (present(p + from, bytes)) fail("untouched pages present");
            if (!des::pages_ready(p + from, bytes, true)) fail("untouched pages refused");
            if (!present(p + from, bytes)) fail("pages not brought in");
            for (size_t i = 0; i < bytes; i += 511)
                if (p[from + i]) return fail("a byte changed"), 1;
            munmap(p, n);
            p = map();
            if (!des::pages_ready(p + from, bytes, false)) fail("untouched pages refused to a reader");
            munmap(p, n);
        }
    char *p = map();
    for (size_t i = 0; i < n / 2; ++i) p[i] = (char)(i * 7);
    madvise(p + n / 4, page, MADV_DONTNEED);         // one page back to zeros
    for (bool write : {false, true}) {
        if (!des::pages_ready(p, n, write)) fail("partly touched pages refused");
        if (write && !present(p, n)) fail("partly touched pages not brought in");
    }
    for (size_t i = 0; i < n; ++i)
        if (p[i] != (i < n / 2 && (i < n / 4 || i >= n / 4 + page) ? (char)(i * 7) : 0)) return fail("a byte changed"), 1;
    struct {
        const char *what;
        char *at;
        int prot;
        bool read, write;
    } const closed[] = {{"first page read-only", p, PROT_READ, true, false},
                        {"last page read-only", p + n - page, PROT_READ, true, false},
                        {"first page closed", p, PROT_NONE, false, false},
                        {"last page closed", p + n - page, PROT_NONE, false, false}};
    for (const auto &c : closed) {
        mprotect(c.at, page, c.prot);
        if (des::pages_ready(p + 8, n - 16, false) != c.read || des::pages_ready(p + 8, n - 16, true) != c.write) fail(c.what);
        if (des::pages_ready(c.at + 8, 16, false) != c.read || des::pages_ready(c.at + 8, 16, true) != c.write) fail(c.what);
        mprotect(c.at, page, PROT_READ | PROT_WRITE);
    }
    munmap(p + n / 2, page);
    if (des::pages_ready(p, n, false) || des::pages_ready(p, n, true)) fail("an unmapped page in the middle");
    if (des::pages_ready(p, n / 2 + 1, false) || des::pages_ready(p, n / 2 + 1, true)) fail("an unmapped page at the end");
    if (!des::pages_ready(p, n / 2, true)) fail("the pages before it");
    printf("%d mismatches\n", bad);
    return bad != 0;
}
