// Host pages of a result buffer, made present before the device writes to it.
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace mnad {

// Fresh host memory (an untouched allocation) is otherwise faulted in by the copy
// from the device: a shot record into a new array took 5.3 ms instead of 1.8 at
// 4 MB, 17.7 instead of 4.8 at 16 MB, 32.5 instead of 8.3 at 30 MB (touching page
// by page 2.2, 6.4 and 11.6), the first download of 16 RTM shots of 481 x 1281
// 57 instead of 8 ms.  Above 32 MB the driver copies with host threads, which
// fault as fast.
constexpr size_t POPULATE_MIN = 256 << 10, POPULATE_MAX = 30 << 20;

// No byte changes, and nothing happens where the range is not mapped.  A buffer
// that is present already (every download after the first) is only looked up:
// populating it again walks its pages, 34 us per 8 MB with pages of 64 KB, the
// look-up 1.3 us.
inline void populate_pages(void* dst, size_t bytes)
{
#ifdef MADV_POPULATE_WRITE
    static const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    if (!dst || bytes < POPULATE_MIN || bytes > POPULATE_MAX) return;
    const uintptr_t a = (uintptr_t)dst / page * page, b = ((uintptr_t)dst + bytes + page - 1) / page * page;
    std::vector<unsigned char> present((b - a) / page);
    if (mincore((void*)a, b - a, present.data()) == 0 &&
        std::all_of(present.begin(), present.end(), [](unsigned char x) { return x & 1; }))
        return;
    madvise((void*)a, b - a, MADV_POPULATE_WRITE);
#else
    (void)dst, (void)bytes;
#endif
}

}  // namespace mnad
