// Host check of pages_present and pages_allow (csrc/des_hostmem.h): untouched,
// touched, partly touched, released, protected and unmapped ranges.  exit 1 on a
// mismatch.
#include "des_hostmem.h"

#include <cstdio>
#include <cstring>

int main()
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = (size_t)64 << 20;
    char *p = static_cast<char *>(mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (p == MAP_FAILED) return 1;
    madvise(p, n, MADV_NOHUGEPAGE);
    int bad = 0;
    auto expect = [&](const char *what, const void *q, size_t bytes, bool want) {
        const bool got = des::pages_present(q, bytes);
        if (got != want) printf("%s: %d\n", what, got), ++bad;
    };
    expect("untouched", p, n, false);
    expect("small, untouched", p, ((size_t)1 << 20) - 1, true);
    std::memset(p, 1, n / 2);
    expect("touched half", p, n / 2, true);
    expect("touched half, off a page", p + 24, n / 2 - 48, true);
    expect("one page more", p, n / 2 + page, false);
    expect("one byte more", p + 8, n / 2 - 7, false);
    std::memset(p, 1, n);
    expect("touched", p, n, true);
    madvise(p + n / 4, page, MADV_DONTNEED);
    expect("one page given back", p, n, false);
    expect("after that page", p + n / 4 + page, n / 2, true);
    munmap(p + n / 2, page);
    expect("one page unmapped", p + n / 4 + page, n / 2, false);
    auto allow = [&](const char *what, const void *q, size_t bytes, bool write, bool want) {
        const bool got = des::pages_allow(q, bytes, write);
        if (got != want) printf("%s, %s: %d\n", what, write ? "write" : "read", got), ++bad;
    };
    char *r = p + n / 4 + page;                      // touched pages up to the unmapped one
    const size_t m = n / 4 - page;
    r[5] = 17;
    for (bool write : {false, true}) {
        allow("ordinary", r, m, write, true);
        allow("a few bytes", r + 3, 40, write, true);
        allow("over a page's end", r + page - 8, 16, write, true);
        allow("into the unmapped page", r, m + 1, write, false);
    }
    mprotect(r, page, PROT_READ);
    allow("first page read-only", r + 8, m - 8, false, true);
    allow("first page read-only", r + 8, m - 8, true, false);
    mprotect(r, page, PROT_READ | PROT_WRITE);
    mprotect(r + m - page, page, PROT_NONE);
    allow("last page closed", r, m, false, false);
    allow("last page closed", r, m, true, false);
    if (r[5] != 17) printf("contents changed\n"), ++bad;
    printf("%d mismatches\n", bad);
    return bad != 0;
}
