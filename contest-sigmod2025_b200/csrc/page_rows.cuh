// Rows and values of a page with NULLs, whose values lie densely: from the null
// bitmap at the page's end and the page index.
#pragma once

#include "device.cuh"

namespace bj {

// Bitmap bits of rows 32 w .. 32 w + 31 of a page whose nbytes bitmap bytes
// end the page (bits beyond the page's rows are garbage).
__device__ __forceinline__ uint32_t page_bitmap_word(const uint8_t* pg, uint32_t nbytes, uint32_t w) {
    const uint32_t byte = kPageSize - nbytes + 4 * w;
    const uint32_t lo = byte & ~3u;
    if (lo >= kPageSize) return 0;
    const uint32_t a = *reinterpret_cast<const uint32_t*>(pg + lo);
    const uint32_t b = lo + 4 < kPageSize ? *reinterpret_cast<const uint32_t*>(pg + lo + 4) : 0u;
    return __funnelshift_r(a, b, 8 * (byte & 3));
}

// Row of value d of a page of n rows, some of them NULL: the 64-row chunk that
// holds the value by the page index (dense: the values before each of its
// chunks), then the bit of the chunk's bitmap. Ends, with some row, for a page
// that contradicts its index or holds values but no rows: the index checks
// pages as they are uploaded, not those of a loaded snapshot.
__device__ __forceinline__ uint32_t row_of_value(const uint8_t* pg, uint32_t n, const uint32_t* dense, uint32_t d) {
    uint32_t lo = 0, hi = n ? (n - 1) / 64 : 0;  // the last chunk with at most d values before it
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) / 2;
        if (__ldg(dense + mid) <= d)
            lo = mid;
        else
            hi = mid - 1;
    }
    uint32_t k = d - __ldg(dense + lo);  // set bits of the chunk before the value's
    const uint32_t nbytes = (n + 7) >> 3;
    uint32_t w = page_bitmap_word(pg, nbytes, 2 * lo), r = 64 * lo;
    if (k >= uint32_t(__popc(w))) {
        k -= __popc(w);
        w = page_bitmap_word(pg, nbytes, 2 * lo + 1);
        r += 32;
    }
    for (; k && w; k--) w &= w - 1;
    return r + (w ? __ffs(w) - 1 : 0);
}

} // namespace bj
