// row_of_value and page_bitmap_word (csrc/page_rows.cuh), compiled for the host: every value of pages of many shapes gets
// its row, and pages that contradict their index end the search too.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline
static long g_loads = 0;  // loads of the index: a search that does not end is stopped here
struct Endless {};
static uint32_t __ldg(const uint32_t* p) {
    if (++g_loads > 1000) throw Endless{};
    return *p;
}
static int __popc(uint32_t w) { return __builtin_popcount(w); }
static int __ffs(uint32_t w) { return __builtin_ffs(int(w)); }
static uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return uint32_t(((uint64_t(hi) << 32) | lo) >> (s & 31));
}

#include "page_rows.cuh"

using bj::kPageSize;

struct PageOf {
    alignas(16) uint8_t bytes[kPageSize] = {};
    uint32_t n = 0;
    std::vector<uint32_t> dense, row;  // the index; row of every value
    PageOf(uint32_t rows, double valid, std::mt19937& rng) : n(rows) {
        const uint32_t nbytes = (n + 7) / 8, most = (kPageSize - 4 - nbytes) / 4;
        for (uint32_t r = 0; r < n; r++) {
            if (r % 64 == 0) dense.push_back(uint32_t(row.size()));
            if (row.size() < most && std::uniform_real_distribution<>()(rng) < valid) {
                bytes[kPageSize - nbytes + r / 8] |= uint8_t(1u << (r % 8));
                row.push_back(r);
            }
        }
        const uint32_t hdr = n | uint32_t(row.size()) << 16;
        std::memcpy(bytes, &hdr, 4);
        // Bits beyond the rows are anything.
        if (n % 8) bytes[kPageSize - 1] |= uint8_t(0xff << (n % 8));
    }
};

int main() {
    std::mt19937 rng(1);
    for (uint32_t n : {1u, 7u, 8u, 31u, 32u, 33u, 63u, 64u, 65u, 127u, 129u, 1000u, 1984u, 2047u, 3072u, 3073u, 20000u, 60001u})
        for (double valid : {0.0, 0.03, 0.5, 0.97, 1.0}) {
            const PageOf p(n, valid, rng);
            for (uint32_t w = 0; w < (n + 31) / 32; w++) {
                uint32_t want = 0;
                for (uint32_t r : p.row)
                    if (r / 32 == w) want |= 1u << (r % 32);
                const uint32_t own = n - 32 * w < 32 ? (1u << (n - 32 * w)) - 1 : ~0u;
                if ((bj::page_bitmap_word(p.bytes, (n + 7) / 8, w) & own) != want) {
                    std::printf("n %u valid %g: bitmap word %u\n", n, valid, w);
                    return 1;
                }
            }
            for (uint32_t d = 0; d < p.row.size(); d++) {
                g_loads = 0;
                const uint32_t got = bj::row_of_value(p.bytes, n, p.dense.data(), d);
                if (got != p.row[d]) {
                    std::printf("n %u valid %g: value %u in row %u, not %u\n", n, valid, d, got, p.row[d]);
                    return 1;
                }
            }
        }
    // Values but no rows; an index of another page; an index of nonsense.
    try {
        const PageOf p(2000, 0.5, rng);
        std::vector<uint32_t> zero(1024, 0), wild(1024, 0xfffffff0u);
        for (uint32_t d : {0u, 1u, 31u, 64u, 2046u})
            for (uint32_t n : {0u, 1u, 64u, 2000u, 65535u})
                for (const auto& index : {zero, wild}) {
                    g_loads = 0;
                    const uint32_t r = bj::row_of_value(p.bytes, n, index.data(), d);
                    if (r >= 65536) {
                        std::printf("row %u of a page that has at most 65,535\n", r);
                        return 1;
                    }
                }
    } catch (const Endless&) {
        std::puts("a search does not end");
        return 1;
    }
    std::puts("ok");
    return 0;
}
