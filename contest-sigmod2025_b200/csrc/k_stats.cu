// Column statistics, exact sub-plan cardinalities and join samples: the
// inputs of join ordering.
//
// The reference estimates cardinalities from 64 sampled rows per base table
// (engine/query/QueryPlan.cpp:719-746, TableScan.cpp:743-772): a row's key is
// tested against the restrictions of its equivalence class, and an input's
// cardinality is its rows times the share of sampled rows that pass
// (QueryPlan.cpp:67-72). The kernels here provide what join ordering needs on
// the device:
//
//  * k_col_stats: per join-key column, a 64-bin histogram of its non-null
//    values by the top six bits of the key hash, and a key -> count map (the
//    index the join samples and exact counts look keys up in);
//  * k_count_node, k_count_group: exact counts of join results, by weights
//    instead of rows (a row's weight is the number of join results it takes
//    part in below it): children's maps are looked up, weights multiplied, and
//    summed into the parent-edge key's map (an inner table), or into the
//    totals of the sub-plans that have the table at their root, so a count
//    never materialises a join result;
//  * k_sample_edges: for every directed join edge, how many of 64 sampled
//    rows of one side find their key in the other side's map (the
//    reference's join sample).
#include "launch.h"

#include <cuda_runtime.h>

namespace bj {
namespace {

constexpr unsigned long long kMapEmpty = ~0ull;

__device__ __forceinline__ uint32_t map_slot(uint64_t key, uint32_t log2cap) {
    return uint32_t(mix64(key) >> (64 - log2cap));
}

// *y += v for v > 0; a sum past 2^64 - 1 stays at ~0ull. Whoever sees the word
// wrap puts it there, and an addition that comes after wraps again and does the
// same, so in any order the last write leaves ~0ull. Returns what was there.
__device__ __forceinline__ unsigned long long add_sat(unsigned long long* y, unsigned long long v) {
    const unsigned long long old = atomicAdd(y, v);
    if (old + v < old) atomicMax(y, ~0ull);
    return old;
}

// Adds v to key's value (inserting the key); returns 1 when the key is new. The
// key ~0ull, which marks empty slots, keeps its value in slot cap.
__device__ __forceinline__ uint32_t map_add(const KeyMap& m, uint64_t key, unsigned long long v, uint32_t* err) {
    const uint32_t cap = 1u << m.log2cap;
    if (key == kMapEmpty) return add_sat(&m.slots[cap].y, v) == 0 ? 1u : 0u;
    uint32_t pos = map_slot(key, m.log2cap), added = 0;
    for (uint32_t step = 0; step < cap; step++) {
        unsigned long long cur = m.slots[pos].x;
        if (cur == kMapEmpty) {
            cur = atomicCAS(&m.slots[pos].x, kMapEmpty, key);
            if (cur == kMapEmpty) {
                added = 1;
                cur = key;
            }
        }
        if (cur == key) {
            add_sat(&m.slots[pos].y, v);
            return added;
        }
        pos = (pos + 1) & (cap - 1);
    }
    record_error(err, kErrCapacity);
    return 0;
}

// Key's value in a finished map (0 when it is not there): key and value in one
// 16-byte load.
__device__ __forceinline__ unsigned long long map_get(const KeyMap& m, uint64_t key) {
    const uint32_t cap = 1u << m.log2cap;
    if (key == kMapEmpty) return m.slots[cap].y;
    uint32_t pos = map_slot(key, m.log2cap);
    for (uint32_t step = 0; step < cap; step++) {
        const ulonglong2 cur = __ldg(m.slots + pos);
        if (cur.x == key) return cur.y;
        if (cur.x == kMapEmpty) return 0;
        pos = (pos + 1) & (cap - 1);
    }
    return 0;
}

__global__ void k_map_clear(KeyMap m) {
    const uint32_t cap = 1u << m.log2cap;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= cap; i += gridDim.x * blockDim.x)
        m.slots[i] = make_ulonglong2(kMapEmpty, 0);
}

// `parts` CTAs per page (grid-stride): a page stores its non-null values
// densely, so the histogram and the map need neither the bitmap nor the row
// index. A column of few pages is split further: its CTAs' chains of atomics
// are what it takes (45K rows in 23 pages: 33 us whole, 13 us in eight parts).
__global__ void __launch_bounds__(256) k_col_stats(DevColumn c, uint32_t parts, KeyMap m, uint32_t* hist,
                                                   unsigned int* totals, uint32_t* err) {
    __shared__ uint32_t h[kHistBins];
    for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint32_t width = c.type == kInt32 ? 4 : 8;
    uint32_t nonnull = 0, distinct = 0;
    for (uint32_t u = blockIdx.x; u < c.npages * parts; u += gridDim.x) {
        const uint32_t p = u / parts;
        const uint8_t* pg = c.pages + size_t(p) * kPageSize;
        const uint32_t hd = c.hdr ? c.hdr[p] : *reinterpret_cast<const uint32_t*>(pg);
        const uint32_t nn = hd >> 16;
        const uint32_t base = width;  // values start at byte 4 (INT32) or 8 (INT64)
        for (uint32_t i = (u % parts) * blockDim.x + threadIdx.x; i < nn; i += parts * blockDim.x) {
            uint64_t key = width == 4 ? uint64_t(*reinterpret_cast<const uint32_t*>(pg + base + 4 * i))
                                      : *reinterpret_cast<const uint64_t*>(pg + base + 8 * size_t(i));
            atomicAdd(&h[key_hash_any(key, c.type) >> 58], 1u);
            distinct += map_add(m, key, 1ull, err);
            nonnull++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        nonnull += __shfl_down_sync(0xffffffffu, nonnull, o);
        distinct += __shfl_down_sync(0xffffffffu, distinct, o);
    }
    if ((threadIdx.x & 31) == 0 && nonnull) atomicAdd(&totals[0], nonnull);
    if ((threadIdx.x & 31) == 0 && distinct) atomicAdd(&totals[1], distinct);
    __syncthreads();
    for (int i = threadIdx.x; i < kHistBins; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], h[i]);
}

// Saturating u64 product: ~0ull stands for a weight past 2^64 - 1 and stays that
// unless the other factor is 0.
__device__ __forceinline__ unsigned long long mul_sat(unsigned long long a, unsigned long long b) {
    return __umul64hi(a, b) ? ~0ull : a * b;
}

// An inner table's map: each row's weight, summed into its parent-edge key.
__global__ void __launch_bounds__(256) k_count_node(CountNode n, uint32_t* err) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n.nrows; r += gridDim.x * blockDim.x) {
        unsigned long long w = 1;
        for (int j = 0; j < n.nch && w; j++) {
            uint64_t k;
            if (!col_get(n.ch[j].key, r, k)) {
                w = 0;
                break;
            }
            w = mul_sat(w, map_get(n.ch[j].map, k));
        }
        if (!w) continue;
        uint64_t k;
        if (col_get(n.pkey, r, k)) map_add(n.out, k, w, err);
    }
}

// The totals of sub-plans with the same root table, in one pass over it. A
// tile's rows look up every option (a child edge with the sub-tree below it
// that some sub-plan has there) once. A row whose options are all 0 or 1 (keys
// unique on the child's side) counts 1 in every total whose options it has, so
// only its set of options is counted, and the sets' counts go into the totals
// at the end; the other rows' options are multiplied, a warp a total, a lane a
// row. The pass, its keys and the lookups' random sectors are paid once for up
// to kMaxCountTotals sub-plans instead of for each.
// The 26 totals over the 1.5M-row root of a seven-table query on a B200: 93
// us, where a pass a total took 26 x 40 us; every row multiplied: 191 us.
// kFew: at most kFewTotals totals, which would leave half of the warps or more to
// wait for the others: a row's own thread multiplies its options, without a barrier, and looks
// no further once one that all totals have is 0. One total of four tables over
// rows that are all multiplied: the call 189 us in the other form, 77 us so. (Eight
// totals are a warp's each: 91 us for the labels of a 500K-row fact in the other
// form, 101 so.)
constexpr int kFewTotals = 4;
template <bool kFew>
__global__ void __launch_bounds__(256) k_count_group(CountGroup g) {
    extern __shared__ uint32_t sets[];  // rows by set of options, 1 << nopt
    __shared__ unsigned long long w[kMaxCountOptions][256];
    __shared__ uint32_t heavy[kFew ? 1 : 256];  // per row: its options when one is above 1, else 0
    constexpr int kPerWarp = kFew ? kFewTotals : kMaxCountTotals / 8;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // Totals i = 0, 1, ... of this warp: number warp + 8 i, or (kFew) its part of number i.
    const auto total_of = [&](int i) { return kFew ? i : int(warp) + 8 * i; };
    unsigned long long acc[kPerWarp] = {};
    uint32_t over = 0;  // bit i: this warp's i-th total passed 2^64 - 1
    const auto add_row = [&](unsigned long long& sum, int i, uint32_t row, uint32_t set) {
        unsigned long long v = 1;
        for (uint32_t m = set; m; m &= m - 1) {
            const unsigned long long x = w[__ffs(m) - 1][row];
            v = (v | x) >> 32 ? mul_sat(v, x) : static_cast<unsigned long long>(uint32_t(v)) * uint32_t(x);
        }
        sum += v;
        if (v == ~0ull || sum < v) over |= 1u << i;
    };
    for (uint32_t m = t; m < 1u << g.nopt; m += 256) sets[m] = 0;
    __syncthreads();
    for (uint32_t r0 = blockIdx.x * 256; r0 < g.nrows; r0 += gridDim.x * 256) {
        const uint32_t r = r0 + t;
        uint64_t key = 0;
        bool ok = false, above = false;
        bool live = r < g.nrows;  // may still be in some total
        uint32_t have = 0;
        for (int o = 0; o < g.nopt; o++) {  // (with one end: lanes that left it earlier would part from the others)
            const CountOption& op = g.opt[o];
            if (op.new_edge) ok = live && col_get(op.key, r, key);
            // A key that the child's own rows lack is in none of its sub-trees' maps.
            const bool gone = (op.leaf >= 0 && !((have >> op.leaf) & 1)) || (kFew && !live);
            const unsigned long long v = ok && !gone ? map_get(op.map, key) : 0ull;
            if (kFew) live = live && (v || !(g.all >> o & 1));
            w[o][t] = v;
            above = above || v > 1;
            if (v) have |= 1u << o;
        }
        if (kFew && !live) have = 0, above = false;
        const uint32_t same = __match_any_sync(0xffffffffu, above ? 0u : have);
        if (!above && have && lane == uint32_t(__ffs(same) - 1)) atomicAdd(&sets[have], __popc(same));
        if (kFew) {
            if (!above) continue;
#pragma unroll
            for (int i = 0; i < kFewTotals; i++)
                if (i < g.ntot && (have & g.options[i]) == g.options[i]) add_row(acc[i], i, t, g.options[i]);
            continue;
        }
        heavy[kFew ? 0 : t] = above ? have : 0u;
        if (!__syncthreads_or(above)) continue;
#pragma unroll
        for (int i = 0; i < kPerWarp; i++) {
            const int s = total_of(i);
            if (s >= g.ntot) continue;
            const uint32_t set = g.options[s];
            for (int j = 0; j < 8; j++)
                if ((heavy[kFew ? 0 : 32 * j + lane] & set) == set) add_row(acc[i], i, 32 * j + lane, set);
        }
        __syncthreads();
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPerWarp; i++) {
        const int s = total_of(i);
        if (s >= g.ntot) continue;
        const uint32_t set = g.options[s];
        unsigned long long v = acc[i];
        bool o1 = (over >> i) & 1;
        if (!kFew || warp == 0)
            for (uint32_t m = lane; m < 1u << g.nopt; m += 32)
                if ((m & set) == set) {
                    const unsigned long long sum = v + sets[m];
                    o1 = o1 || sum < v;
                    v = sum;
                }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
            o1 = o1 || v + u < v;
            v += u;
        }
        o1 = __any_sync(0xffffffffu, o1);
        if (lane == 0 && v) {
            const unsigned long long old = atomicAdd(g.total + g.slot[s], v);
            o1 = o1 || old + v < old;
        }
        if (lane == 0 && o1) atomicOr(g.flags + 2 * g.slot[s], 1u);
    }
}

// Row i of a sample: a seeded position (the reference samples 64 rows with
// its own seeded generator, engine/infra/Random.hpp:7-29).
__global__ void k_sample_edges(SampleEdges e, uint32_t nsample, uint32_t* hits) {
    const int d = blockIdx.x;
    if (d >= e.n) return;
    const SampleEdge& s = e.e[d];
    uint32_t mine = 0;
    for (uint32_t i = threadIdx.x; i < nsample && s.key.nrows; i += blockDim.x) {
        const uint32_t row = uint32_t(mix64(0x5a17ull * (d + 1) + i + (uint64_t(s.seed) << 32)) % s.key.nrows);
        uint64_t k;
        if (col_get(s.key, row, k) && map_get(s.map, k) != 0) mine++;
    }
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&hits[d], mine);
}

} // namespace

int map_clear(const KeyMap& m, cudaStream_t st) {
    const uint32_t cap = 1u << m.log2cap;
    const uint32_t blocks = std::min<uint32_t>((cap + 256) / 256, 148 * 8);
    k_map_clear<<<blocks, 256, 0, st>>>(m);
    return 1;
}

int column_stats(const DevColumn& c, const KeyMap& m, uint32_t* hist, unsigned int* totals, uint32_t* err, int num_sms,
                 cudaStream_t st) {
    if (!c.npages) return 0;
    const uint32_t most = uint32_t(num_sms) * 8, parts = std::min<uint32_t>(8, std::max<uint32_t>(1, most / c.npages));
    k_col_stats<<<std::min<uint32_t>(c.npages * parts, most), 256, 0, st>>>(c, parts, m, hist, totals, err);
    return 1;
}

int count_node(const CountNode& n, uint32_t* err, int num_sms, cudaStream_t st) {
    if (!n.nrows) return 0;
    const uint32_t blocks = std::min<uint32_t>((n.nrows + 255) / 256, uint32_t(num_sms) * 8);
    k_count_node<<<blocks, 256, 0, st>>>(n, err);
    return 1;
}

int count_group(const CountGroup& g, int num_sms, cudaStream_t st) {
    if (!g.nrows || !g.ntot) return 0;
    const uint32_t blocks = std::min<uint32_t>((g.nrows + 255) / 256, uint32_t(num_sms) * 8);
    const size_t sets = sizeof(uint32_t) << g.nopt;
    g.ntot <= kFewTotals ? k_count_group<true><<<blocks, 256, sets, st>>>(g) : k_count_group<false><<<blocks, 256, sets, st>>>(g);
    return 1;
}

int sample_edges(const SampleEdges& e, uint32_t nsample, uint32_t* hits, cudaStream_t st) {
    if (!e.n) return 0;
    k_sample_edges<<<e.n, 64, 0, st>>>(e, nsample, hits);
    return 1;
}

} // namespace bj
