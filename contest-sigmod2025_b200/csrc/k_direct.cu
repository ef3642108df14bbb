// K2 + K3 + K5, second form: the scan-side probe without a staged filter.
//
// k_scan.cu gives a warp 4 KiB of keys and a CTA a 128 KiB filter: right for
// long scans of a selective probe, where the filter keeps most rows from ever
// touching the table. Two kinds of scan want neither (TableScan::produceImpl
// and HashtableProbe, engine/op/TableScan.cpp:616-741, Hashtable.hpp:228-241):
// a probe that most rows pass (or a column with NULLs, whose rows that form
// takes one by one), and a table of a few hundred pages, which there runs on
// a handful of warps, each working through a long chain of dependent loads.
//
// Here a CTA of 256 threads takes a page, or an eighth, quarter or half of one
// where pages are few. Lane l of a warp has row l of a
// group of 32 rows, so keys, items and the null bitmap are read and written
// coalesced, and four groups at a time are probed with their bucket loads in
// flight together. Matches leave in one append (one global atomic a page),
// from the registers that found them, or, when unique-key stages follow the
// scan, from shared memory after those stages ran on them (JoinPipeline.hpp:
// 111-131 fuses the same stages), which saves their launch and the items
// between.
//
// Bound: the bucket lookups' L2 sectors (8M probes of a 1M-key table: 58 us,
// 136 G sectors/s), below a few thousand pages the latency of one page.
// Measured on a B200 against the staged form, device time of the scan (with
// the stages after it): 30K rows in 16 pages 30 -> 10 us; 1M rows, two tables
// 28 -> 16 us; 8M rows with 10% NULLs 145 -> 63 us (75 us with the matches
// staged in shared memory and 1,184 CTAs looping over the pages).
#include "launch.h"
#include "page_rows.cuh"

#include <algorithm>

namespace bj {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kGroups = 4;             // groups of 32 rows probed together by a warp
constexpr uint32_t kPageValues = 2048; // more than the values of any page
constexpr uint32_t kMaxParts = 8;      // blocks a page at most

struct DirectArgs {
    DevColumn key;
    HTView ht;
    uint32_t use_bloom;  // test ht.bloom (in global memory) before the bucket
    uint32_t parts;      // blocks a page
    ProbeChain chain;
    ItemsOut out;
    uint32_t* cursor;
    uint32_t capacity;
    uint32_t* err;
};

template <bool kWide>
__device__ __forceinline__ uint64_t load_value(const uint8_t* pg, uint32_t d) {
    if (kWide) return __ldg(reinterpret_cast<const unsigned long long*>(pg + 8) + d);
    return __ldg(reinterpret_cast<const uint32_t*>(pg + 4) + d);
}

// The entry each of a lane's kGroups keys matches (unique keys: at most one).
// `valid` flags the keys present; the result flags the matches in e.
template <bool kWide>
__device__ __forceinline__ uint32_t probe_groups(const DirectArgs& a, const uint64_t (&key)[kGroups], uint32_t valid,
                                                 uint32_t (&e)[kGroups]) {
    const HTView& ht = a.ht;
    if (!kWide && a.use_bloom) {
#pragma unroll
        for (int k = 0; k < kGroups; k++)
            if (((valid >> k) & 1) && !bloom_may_contain(ht.bloom, ht.bloom_log2, uint32_t(key[k]))) valid &= ~(1u << k);
    }
    uint4 b[kGroups];
#pragma unroll
    for (int k = 0; k < kGroups; k++) {
        b[k] = make_uint4(0, 0, 0, 0);
        if ((valid >> k) & 1) b[k] = __ldg(ht.buckets + bucket_of(key[k], kWide, ht.shift));
    }
    uint32_t hit = 0;
#pragma unroll
    for (int k = 0; k < kGroups; k++) {
        e[k] = 0;
        if (!kWide) {
            const uint32_t kk = uint32_t(key[k]);
            const bool first = b[k].y >= 1 && b[k].z == kk, second = b[k].y >= 2 && b[k].w == kk;
            e[k] = b[k].x + (second ? 1u : 0u);
            if (first || second) hit |= 1u << k;
        }
    }
#pragma unroll
    for (int k = 0; k < kGroups; k++) {
        if ((hit >> k) & 1) continue;
        if (kWide) {
            bucket_matches(ht, b[k], key[k], [&](uint32_t j) {
                e[k] = j;
                hit |= 1u << k;
                return false;
            });
        } else {
            // Buckets of three entries and more.
            for (uint32_t j = 2; j < b[k].y; j++)
                if (uint32_t(ht_key(ht, b[k].x + j)) == uint32_t(key[k])) {
                    e[k] = b[k].x + j;
                    hit |= 1u << k;
                    break;
                }
        }
    }
    return hit;
}

// First entry of `ht` with this key (unique keys), or false.
__device__ __forceinline__ bool find_entry(const HTView& ht, uint64_t key, bool use_bloom, uint32_t& e) {
    if (use_bloom && ht.bloom && !bloom_may_contain(ht.bloom, ht.bloom_log2, uint32_t(key))) return false;
    bool found = false;
    bucket_matches(ht, ht_bucket(ht, key), key, [&](uint32_t j) {
        e = j;
        found = true;
        return false;
    });
    return found;
}

// A page's shape: rows, whether some are NULL, its first row and chunk.
struct PageShape {
    uint32_t n, row0, chunk0;
    bool nulls;
};
__device__ __forceinline__ PageShape page_shape(const DevColumn& c, uint32_t p) {
    const uint32_t hdr = __ldg(reinterpret_cast<const uint32_t*>(c.pages + size_t(p) * kPageSize));
    PageShape s;
    s.n = hdr & 0xffff;
    s.nulls = (hdr >> 16) != s.n;
    s.row0 = c.rpp ? p * c.rpp : __ldg(c.row_start + p);
    s.chunk0 = s.nulls ? __ldg(c.chunk_base + p) : 0u;
    return s;
}

// This block's rows of its page: [first, end), first a multiple of 64; empty
// beyond the page's rows.
__device__ __forceinline__ void block_rows(const DirectArgs& a, const PageShape& s, uint32_t& first, uint32_t& end) {
    const uint32_t span = (s.n + 64 * a.parts - 1) / (64 * a.parts) * 64;
    first = blockIdx.x % a.parts * span;
    end = min(first + span, s.n);
}

// The keys of kGroups groups of 32 rows of a page from row r0 (a multiple of
// 64, below `end`), a row a lane, none at or beyond row `end`; the result
// flags the lanes' rows that have one.
template <bool kWide>
__device__ __forceinline__ uint32_t load_groups(const DirectArgs& a, const uint8_t* pg, const PageShape& s, uint32_t r0,
                                                uint32_t end, uint64_t (&key)[kGroups]) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t valid = 0;
    if (!s.nulls) {
#pragma unroll
        for (int k = 0; k < kGroups; k++) {
            const uint32_t r = r0 + 32 * k + lane;
            key[k] = 0;
            if (r < end) {
                key[k] = load_value<kWide>(pg, r);
                valid |= 1u << k;
            }
        }
        return valid;
    }
    // The value index of a row comes from the page index and the bitmap.
    uint32_t word = 0;
    if (lane < kGroups && r0 + 32 * lane < end) {
        word = page_bitmap_word(pg, (s.n + 7) >> 3, r0 / 32 + lane);
        const uint32_t left = end - (r0 + 32 * lane);
        if (left < 32) word &= (1u << left) - 1;
    }
    uint32_t dense = __ldg(a.key.dense_base + s.chunk0 + (r0 >> 6));
#pragma unroll
    for (int k = 0; k < kGroups; k++) {
        const uint32_t w = __shfl_sync(0xffffffffu, word, k);
        const uint32_t d = dense + __popc(w & ((1u << lane) - 1));
        dense += __popc(w);
        key[k] = 0;
        if (((w >> lane) & 1) && d < kPageValues) {
            key[k] = load_value<kWide>(pg, d);
            valid |= 1u << k;
        }
    }
    return valid;
}

// The scan alone: a warp keeps its rows' matches in registers until the block
// has reserved the page's items, and writes them in place.
template <bool kWide>
__global__ void __launch_bounds__(kThreads, 5) k_scan_direct(DirectArgs a) {
    constexpr int kRounds = 3;  // rounds of kGroups groups a warp holds
    __shared__ uint32_t count[kWarps], base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1;
    const uint32_t p = blockIdx.x / a.parts;
    const uint8_t* pg = a.key.pages + size_t(p) * kPageSize;
    const PageShape s = page_shape(a.key, p);
    uint32_t from, to;
    block_rows(a, s, from, to);
    if (from >= to) return;
    // Rows a warp, in chunks of 64: 256 on a full page without NULLs, more on
    // one with; more than 3,072 rows take several turns.
    const uint32_t share = min((to - from + 64 * kWarps - 1) / (64 * kWarps) * 64, uint32_t(kRounds * kGroups * 32));
    for (uint32_t span = from; span < to; span += share * kWarps) {
        const uint32_t first = span + warp * share, end = min(first + share, to);
        uint32_t e[kRounds][kGroups], hit[kRounds], total = 0;
#pragma unroll
        for (int h = 0; h < kRounds; h++) {
            const uint32_t r0 = first + h * (kGroups * 32);
            hit[h] = 0;
            if (r0 >= end) continue;
            uint64_t key[kGroups];
            const uint32_t valid = load_groups<kWide>(a, pg, s, r0, end, key);
            hit[h] = probe_groups<kWide>(a, key, valid, e[h]);
        }
#pragma unroll
        for (int h = 0; h < kRounds; h++) total += __popc(hit[h]);
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if (lane == 0) count[warp] = total;
        __syncthreads();
        uint32_t o = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            if (w == int(warp)) o = all;
            all += count[w];
        }
        if (threadIdx.x == 0 && all) base = atomicAdd(a.cursor, all);
        __syncthreads();  // (also before count is written again)
        if (!all) continue;  // no items were reserved: base is not this turn's
        o += base;
        if (base + all > a.capacity || base + all < all) {
            if (threadIdx.x == 0) record_error(a.err, kErrCapacity);
            return;
        }
#pragma unroll
        for (int h = 0; h < kRounds; h++) {
            if (first + h * (kGroups * 32) >= end) continue;
#pragma unroll
            for (int k = 0; k < kGroups; k++) {
                const bool mine = (hit[h] >> k) & 1;
                const uint32_t m = __ballot_sync(0xffffffffu, mine);
                if (mine) {
                    const uint32_t at = o + __popc(m & below);
                    a.out.rows[at] = s.row0 + first + (h * kGroups + k) * 32 + lane;
                    a.out.ents[0][at] = e[h][k];
                    if (a.out.mult) a.out.mult[at] = ht_mult(a.ht, e[h][k]);
                }
                o += __popc(m);
            }
        }
    }
}

// The scan with the stages after it: a page's matches collect in shared
// memory, then each takes its further probes.
template <bool kWide>
__global__ void __launch_bounds__(kThreads, 6) k_scan_chain(DirectArgs a) {
    __shared__ uint2 found[kPageValues];  // (row, entry) of the page's matches
    __shared__ uint32_t nfound, base, nkept[2];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1;
    const uint32_t p = blockIdx.x / a.parts;
    if (threadIdx.x == 0) nfound = 0;
    __syncthreads();
    const uint8_t* pg = a.key.pages + size_t(p) * kPageSize;
    const PageShape s = page_shape(a.key, p);
    uint32_t from, to;
    block_rows(a, s, from, to);
    if (from >= to) return;
    const uint32_t share = to - from <= 64 * kWarps ? 64u : 32u * kGroups;  // rows a warp
    for (uint32_t r0 = from + warp * share; r0 < to; r0 += kWarps * share) {
        uint64_t key[kGroups];
        uint32_t e[kGroups];
        const uint32_t valid = load_groups<kWide>(a, pg, s, r0, min(r0 + share, to), key);
        const uint32_t hit = probe_groups<kWide>(a, key, valid, e);
        uint32_t m[kGroups], total = 0;
#pragma unroll
        for (int k = 0; k < kGroups; k++) {
            m[k] = __ballot_sync(0xffffffffu, (hit >> k) & 1);
            total += __popc(m[k]);
        }
        if (!total) continue;
        uint32_t o = 0;
        if (lane == 0) o = atomicAdd(&nfound, total);
        o = __shfl_sync(0xffffffffu, o, 0);
#pragma unroll
        for (int k = 0; k < kGroups; k++) {
            if ((hit >> k) & 1) found[o + __popc(m[k] & below)] = make_uint2(s.row0 + r0 + 32 * k + lane, e[k]);
            o += __popc(m[k]);
        }
    }
    __syncthreads();
    const uint32_t cnt = nfound;
    for (uint32_t i0 = 0, turn = 0; i0 < cnt; i0 += kThreads, turn ^= 1) {
        if (threadIdx.x == 0) nkept[turn] = 0;
        __syncthreads();
        const uint32_t i = i0 + threadIdx.x;
        bool hit = i < cnt;
        const uint2 f = hit ? found[i] : make_uint2(0, 0);
        uint32_t e[kMaxChain];
#pragma unroll
        for (int t = 0; t < kMaxChain; t++) {
            e[t] = 0;
            if (t >= a.chain.n || !hit) continue;
            const ChainStage& c = a.chain.st[t];
            uint64_t v = 0;
            if (c.src.stage >= 0) {  // the scan's own match (stage 0)
                hit = !ht_slot_null(c.src.ht, f.y, c.src.slot);
                if (hit) v = ht_slot(c.src.ht, f.y, c.src.slot);
            } else if (f.x >= c.key.nrows) {
                record_error(a.err, kErrRowRange);
                hit = false;
            } else {
                hit = col_get(c.key, f.x, v);
            }
            hit = hit && find_entry(c.ht, v, c.use_bloom != 0, e[t]);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        uint32_t o = 0;
        if (lane == 0 && m) o = atomicAdd(&nkept[turn], __popc(m));
        o = __shfl_sync(0xffffffffu, o, 0) + __popc(m & below);
        __syncthreads();
        if (threadIdx.x == 0 && nkept[turn]) base = atomicAdd(a.cursor, nkept[turn]);
        __syncthreads();
        if (!hit) continue;
        o += base;
        if (o >= a.capacity) {
            record_error(a.err, kErrCapacity);
            continue;
        }
        a.out.rows[o] = f.x;
        a.out.ents[0][o] = f.y;
        uint64_t mult = ht_mult(a.ht, f.y);
#pragma unroll
        for (int t = 0; t < kMaxChain; t++) {
            if (t >= a.chain.n) continue;
            a.out.ents[1 + t][o] = e[t];
            if (a.out.mult) mult *= ht_mult(a.chain.st[t].ht, e[t]);
        }
        if (a.out.mult) a.out.mult[o] = mult;
    }
}

} // namespace

int scan_probe_direct(const DevColumn& key, const HTView& ht, bool use_bloom, const ProbeChain* chain,
                      const ItemsOut& out, uint32_t* cursor, uint32_t capacity, uint32_t* err, int num_sms,
                      cudaStream_t st) {
    if (!key.npages) return 0;
    DirectArgs a{};
    a.key = key;
    a.ht = ht;
    a.use_bloom = use_bloom && ht.bloom ? 1u : 0u;
    a.out = out;
    a.cursor = cursor;
    a.capacity = capacity;
    a.err = err;
    if (chain) a.chain = *chain;
    // Few pages: several blocks a page while all are resident together (six an
    // SM), since a block's warps take their rows, and its matches their stages,
    // one after another. The scan of 30K rows with one stage after it 26 -> 18
    // us; at 445 pages and more a block has a page, as its atomic and header
    // then cost more than the rows it shares.
    a.parts = kMaxParts;
    while (a.parts > 1 && uint64_t(key.npages) * a.parts > uint64_t(num_sms) * 6) a.parts /= 2;
    const uint32_t blocks = key.npages * a.parts;
    const bool wide = key.type == kInt64;
    if (chain && chain->n > 0)
        wide ? k_scan_chain<true><<<blocks, kThreads, 0, st>>>(a) : k_scan_chain<false><<<blocks, kThreads, 0, st>>>(a);
    else
        wide ? k_scan_direct<true><<<blocks, kThreads, 0, st>>>(a) : k_scan_direct<false><<<blocks, kThreads, 0, st>>>(a);
    return 1;
}

} // namespace bj
