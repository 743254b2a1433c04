// Pages made ahead of a copy: built without CUDA, so a thread that runs this code cannot touch a device.
#include "pages.h"

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

using namespace b200;

static int failed = 0;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); failed = 1; } } while (0)

static char *map(size_t bytes)
{
    void *p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) exit(2);
    madvise(p, bytes, MADV_NOHUGEPAGE);   // a page is a page
    return static_cast<char *>(p);
}
static size_t resident(const char *p, size_t bytes)
{
    const size_t page = sysconf(_SC_PAGESIZE), n = (bytes + page - 1) / page;
    std::vector<unsigned char> in(n);
    if (mincore(const_cast<char *>(p), bytes, in.data()) != 0) exit(2);
    size_t k = 0;
    for (unsigned char c : in) k += c & 1;
    return k;
}

int main()
{
    const size_t page = sysconf(_SC_PAGESIZE), bytes = (size_t)4 << 20, pages = bytes / page;
    std::atomic<bool> go{false}, stop{true};
#ifdef MADV_POPULATE_WRITE
    char *probe = map(page);
    const bool can = madvise(probe, page, MADV_POPULATE_WRITE) == 0;
#else
    const bool can = false;
#endif
    {   // whole pages of a buffer, not its neighbours; contents stay
        char *p = map(bytes);
        memset(p + 5 * page, 7, 3 * page);
        populate_pages(p + 100, bytes - 200, go);
        CHECK(!can || resident(p, bytes) == pages - 2);
        for (size_t k = 0; k < bytes; k++) if (p[k] != (k >= 5 * page && k < 8 * page ? 7 : 0)) { CHECK(!"contents"); break; }
    }
    {   // stopped before it begins; too small; too large; none
        char *p = map(kPopulateEnd);
        populate_pages(p, bytes, stop);
        populate_pages(p, kPopulateMin - 1, go);
        populate_pages(p, kPopulateEnd, go);
        populate_pages(nullptr, bytes, go);
        CHECK(resident(p, kPopulateEnd) == 0);
    }
    {   // memory that cannot be written to is left alone
        char *p = map(bytes);
        mprotect(p, bytes, PROT_READ);
        populate_pages(p, bytes, go);
        CHECK(resident(p, bytes) == 0);
    }
    {   // the thread: both buffers or as far as it came, ended by end() and by the destructor
        char *a = map(bytes), *b = map(bytes);
        PagesAhead ahead;
        CHECK(!ahead.started());
        ahead.start(a, b, bytes);
        CHECK(ahead.started());
        for (int k = 0; can && k < 10000 && resident(b, bytes) < pages; k++) usleep(1000);
        ahead.end();
        CHECK(!ahead.started() && (!can || (resident(a, bytes) == pages && resident(b, bytes) == pages)));
        for (size_t k = 0; k < bytes; k++) if (a[k] || b[k]) { CHECK(!"contents"); break; }
        ahead.start(nullptr, nullptr, bytes);
        ahead.start(a, b, kPopulateMin - 1);
        CHECK(!ahead.started());
        memset(a, 1, bytes);
        memset(b, 1, bytes);
        CHECK(pages_missing(a, bytes) == 0 && pages_missing(b + 1, bytes - 1) == 0);
        ahead.start(a, b, bytes);   // nothing left to do
        CHECK(!ahead.started());
        // a few missing in the middle, and more of them
        char *holes = map(kPopulateEnd);
        memset(holes, 1, kPopulateEnd);
        madvise(holes + 2000 * page, kPagesWorthAThread * page, MADV_DONTNEED);
        CHECK(pages_missing(holes, kPopulateEnd - 1) == kPagesWorthAThread && pages_missing(holes + 1, bytes) == 0);
        ahead.start(a, holes + 2001 * page, bytes);
        CHECK(!ahead.started());
        ahead.start(a, holes + 2000 * page - 1, bytes);
        CHECK(ahead.started());
        ahead.end();
        for (int k = 0; k < 50; k++) {
            PagesAhead other;
            other.start(map(bytes), nullptr, bytes);
        }
    }
    return failed;
}
