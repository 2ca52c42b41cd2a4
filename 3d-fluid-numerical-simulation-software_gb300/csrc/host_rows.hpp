// Checks of the caller's memory before the device reads it.
#pragma once
#include <cstddef>
#include <cstdint>
#include <unistd.h>

namespace gbt {

// Reads a value of every page of [p, p + bytes) on the host, so that a wrong pointer or count, or a page that is not
// mapped or not readable, ends here and not in a kernel that reads the range. What the caller unmaps while
// the call runs is not seen. (1024 pages of 64 KB, 262144 rows of 64 floats: 2 to 10 us.)
inline void read_every_page(const void *p, size_t bytes)
{
    if (bytes == 0) return;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = (uintptr_t)p, last = a + bytes - 1;
    (void)*(const volatile char *)a;
    for (uintptr_t q = (a / page + 1) * page; q <= last && q > a; q += page) (void)*(const volatile char *)q;
}

// Whether a kernel may read the caller's FP32 rows at p where they lie: the device reaches the host's memory (reaches), the
// rows are there (host), and p is aligned, which a copy does not need and a kernel's load does.
inline bool rows_in_place(const void *p, bool reaches, bool host)
{
    return reaches && host && (uintptr_t)p % alignof(float) == 0;
}

}  // namespace gbt
