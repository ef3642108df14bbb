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
// Here a CTA of 256 threads takes a page. Lane l of a warp has row l of a
// group of 32 rows, so keys, items and the null bitmap are read and written
// coalesced, and four groups at a time are probed with their bucket loads in
// flight together. Matches collect in shared memory and leave in one append
// (one global atomic a page). The unique-key stages that follow the scan run
// on the collected rows before they leave (JoinPipeline.hpp:111-131 fuses the
// same stages), which saves their launch and the items between.
//
// Bound: the bucket lookups' L2 sectors (8M probes of a 1M-key table: 67 us),
// below a few thousand pages the latency of one page. Measured on a B200
// against the staged form, device time of the scan (with the stages after
// it): 30K rows in 16 pages 30 -> 10 us; 1M rows, two tables 28 -> 16 us; 8M
// rows with 10% NULLs 145 -> 75 us.
#include "launch.h"

#include <algorithm>

namespace bj {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kGroups = 4;             // groups of 32 rows probed together by a warp
constexpr uint32_t kPageValues = 2048; // more than the values of any page

struct DirectArgs {
    DevColumn key;
    HTView ht;
    uint32_t use_bloom;  // test ht.bloom (in global memory) before the bucket
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

// Bitmap bits of rows 32 w .. 32 w + 31 of a page whose nbytes bitmap bytes
// end the page (bits beyond the page's rows are garbage).
__device__ __forceinline__ uint32_t bitmap_word(const uint8_t* pg, uint32_t nbytes, uint32_t w) {
    const uint32_t byte = kPageSize - nbytes + 4 * w;
    const uint32_t lo = byte & ~3u;
    if (lo >= kPageSize) return 0;
    const uint32_t a = *reinterpret_cast<const uint32_t*>(pg + lo);
    const uint32_t b = lo + 4 < kPageSize ? *reinterpret_cast<const uint32_t*>(pg + lo + 4) : 0u;
    return __funnelshift_r(a, b, 8 * (byte & 3));
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

template <bool kWide, bool kChain>
__global__ void __launch_bounds__(kThreads, 6) k_scan_direct(DirectArgs a) {
    __shared__ uint2 found[kPageValues];  // (row, entry) of the page's matches
    __shared__ uint32_t nfound, base, nkept[2];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1;
    for (uint32_t p = blockIdx.x; p < a.key.npages; p += gridDim.x) {
        if (threadIdx.x == 0) nfound = 0;
        __syncthreads();
        const uint8_t* pg = a.key.pages + size_t(p) * kPageSize;
        const uint32_t hdr = __ldg(reinterpret_cast<const uint32_t*>(pg));
        const uint32_t n = hdr & 0xffff, nn = hdr >> 16;
        const uint32_t row0 = a.key.rpp ? p * a.key.rpp : __ldg(a.key.row_start + p);
        const uint32_t nbytes = (n + 7) >> 3;
        const uint32_t cb = nn != n ? __ldg(a.key.chunk_base + p) : 0u;
        for (uint32_t r0 = warp * (32 * kGroups); r0 < n; r0 += kWarps * 32 * kGroups) {
            uint64_t key[kGroups];
            uint32_t e[kGroups], valid = 0;
            uint32_t word = 0, dense = r0;
            if (nn != n) {
                // Rows with NULLs before them: the value index comes from the
                // page index (r0 is a multiple of 64) and the bitmap.
                if (lane < kGroups) word = bitmap_word(pg, nbytes, r0 / 32 + lane);
                dense = __ldg(a.key.dense_base + cb + (r0 >> 6));
            }
#pragma unroll
            for (int k = 0; k < kGroups; k++) {
                key[k] = 0;
                uint32_t d = dense + lane;
                bool ok = r0 + 32 * k + lane < n;
                if (nn != n) {
                    uint32_t w = __shfl_sync(0xffffffffu, word, k);
                    const uint32_t left = n - min(n, r0 + 32 * k);
                    if (left < 32) w &= (1u << left) - 1;
                    ok = (w >> lane) & 1;
                    d = dense + __popc(w & below);
                    dense += __popc(w);
                } else {
                    dense += 32;
                }
                if (ok && d < kPageValues - 1) {
                    key[k] = load_value<kWide>(pg, d);
                    valid |= 1u << k;
                }
            }
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
                if ((hit >> k) & 1) found[o + __popc(m[k] & below)] = make_uint2(row0 + r0 + 32 * k + lane, e[k]);
                o += __popc(m[k]);
            }
        }
        __syncthreads();
        const uint32_t cnt = nfound;
        if (!kChain) {
            if (threadIdx.x == 0 && cnt) base = atomicAdd(a.cursor, cnt);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < cnt; i += kThreads) {
                const uint32_t o = base + i;
                if (o >= a.capacity) {
                    record_error(a.err, kErrCapacity);
                    break;
                }
                const uint2 f = found[i];
                a.out.rows[o] = f.x;
                a.out.ents[0][o] = f.y;
                if (a.out.mult) a.out.mult[o] = ht_mult(a.ht, f.y);
            }
            __syncthreads();  // `found` and `nfound` are reused
        } else {
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
            __syncthreads();
        }
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
    const uint32_t blocks = std::min<uint32_t>(key.npages, uint32_t(num_sms) * 8);
    const bool wide = key.type == kInt64, fused = chain && chain->n > 0;
    if (wide)
        fused ? k_scan_direct<true, true><<<blocks, kThreads, 0, st>>>(a)
              : k_scan_direct<true, false><<<blocks, kThreads, 0, st>>>(a);
    else
        fused ? k_scan_direct<false, true><<<blocks, kThreads, 0, st>>>(a)
              : k_scan_direct<false, false><<<blocks, kThreads, 0, st>>>(a);
    return 1;
}

} // namespace bj
