// K3/K4/K6: hash-table build.
//
// The reference builds a chaining table per partition: tuples are appended to
// per-thread chunks (HashtableBuild::operator(), engine/op/Hashtable.hpp:
// 176-203), then every partition is inserted bucket-head first, setting a
// 16-bit bloom word per bucket and folding a tuple into the bucket head when
// key and payload are equal (eager aggregation, engine/op/Hashtable.cpp:
// 208-263). Sizing: 2^max(bit_width(n), 4) buckets (Hashtable.cpp:94-104).
//
// On the GPU the build is a counting sort by bucket. Counting a row into its
// bucket also gives its rank there (the atomic's return value), so the pass
// that places the rows needs no second atomic; a bucket's range may lie
// anywhere, so a block takes the ranges of its 1024 buckets with one atomic
// instead of a device-wide prefix sum. The same bucket index as the
// reference: key_hash(key) >> shift. The blocked bloom filter (K3) is set in
// the counting pass; it is at most 128 KiB so scans can stage it in shared
// memory, and probes consult it before touching the buckets.
//
//  * A leaf (an input that probes nothing) places its rows straight from the
//    column pages: nothing is written between the passes but the ranks. When
//    all leaves of a query are small, one launch builds them, a cluster of
//    CTAs each (k_leaf_cluster).
//  * A build fed by probes writes its tuples first (key, NULL mask, payload,
//    multiplicity), then folds equal ones (eager aggregation, K6) in the next
//    launch: each tuple's index goes into an open-addressing table keyed by
//    the whole tuple. The first copy of each distinct tuple claims a slot with
//    atomicCAS, becomes its representative and counts itself into its bucket;
//    every other copy adds its multiplicity to the representative. Unlike the
//    reference, which only merges with the current bucket head, this folds
//    every duplicate. Builds whose tuples cannot repeat (BuildArgs::distinct)
//    count in the emit and skip the aggregation launch.
//  * The flags of the finished table (repeated keys, multiplicities above 1)
//    come from one pass over the buckets.
// Every buffer that must start at zero is cleared by one memset per build.
//
// Bound: the random sectors of the counts, buckets and entries in L2. The leaf
// of 1M rows with one INT64 payload column, count + ranges + place: 55 us,
// where writing the tuples first, an ordered prefix sum and a scatter into
// separate key, multiplicity, NULL mask and payload arrays took 81 us.
#include "launch.h"

#include <cooperative_groups.h>

#include <algorithm>

namespace bj {
namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ uint64_t tuple_hash(const TupleBuf& t, uint32_t i) {
    uint64_t h = mix64(t.keys[i]);
    if (t.pnull) h = mix64(h ^ t.pnull[i]);
    const uint64_t* p = t.pay + size_t(i) * t.width;
    for (uint32_t j = 0; j < t.width; j++) h = mix64(h ^ (p[j] + 0x9E3779B97F4A7C15ull * (j + 1)));
    return h;
}

// Tuple a (written by another thread, read through L2) equals tuple b.
__device__ __forceinline__ bool tuple_equal_cg(const TupleBuf& t, uint32_t a, uint32_t b) {
    if (__ldcg(t.keys + a) != t.keys[b]) return false;
    if (t.pnull && __ldcg(t.pnull + a) != t.pnull[b]) return false;
    const uint64_t* pa = t.pay + size_t(a) * t.width;
    const uint64_t* pb = t.pay + size_t(b) * t.width;
    for (uint32_t j = 0; j < t.width; j++)
        if (__ldcg(pa + j) != pb[j]) return false;
    return true;
}

// Counts key kv into its bucket and the filter; returns 1 + its rank there.
__device__ __forceinline__ uint32_t count_key(uint32_t* counts, const HTView& ht, uint32_t* bloom, uint64_t kv) {
    if (bloom) {  // INT32 keys only (INT64 tables are built without a filter)
        const uint32_t hh = key_hash_hi(uint32_t(kv));
        atomicOr(&bloom[bloom_word_hi(hh, ht.bloom_log2)], bloom_bits_fast(hh, hh >> 5));
    }
    return 1 + atomicAdd(&counts[bucket_of(kv, ht.wide != 0, ht.shift)], 1u);
}

// Where the entry of key kv with this rank goes in a table whose buckets have
// their ranges; the bucket's first two keys are written into it. False, with
// an error, past the table's end.
__device__ __forceinline__ bool place_key(const HTView& ht, uint64_t kv, uint32_t rank, uint32_t* err, uint32_t& pos) {
    uint4* b = const_cast<uint4*>(ht.buckets) + bucket_of(kv, ht.wide != 0, ht.shift);
    pos = __ldcg(&b->x) + rank;  // (another SM may have written it in this launch)
    if (pos >= ht.nentries) {
        record_error(err, kErrCapacity);
        return false;
    }
    if (rank == 0) b->z = uint32_t(kv);
    if (rank == 1) b->w = uint32_t(kv);
    const_cast<uint64_t*>(ht.ent)[size_t(pos) * (1 + ht.width)] = kv;
    return true;
}

// Eager aggregation of tuple i (every tuple written by an earlier launch):
// the first copy of a distinct tuple to claim a slot of the open-addressing
// table keyed by the whole tuple represents it and is counted into its
// bucket; every other copy adds its multiplicity to the representative.
__device__ __forceinline__ void aggregate_tuple(const BuildArgs& a, uint32_t i) {
    const TupleBuf& t = a.tb;
    const uint64_t m = t.mult[i];  // only a representative's grows, after it claimed its slot
    if (m == 0) return;
    const uint32_t mask = (1u << a.tlog2) - 1;
    uint32_t pos = uint32_t(tuple_hash(t, i) >> (64 - a.tlog2)) & mask;
    for (uint32_t step = 0; step <= mask; step++) {
        const uint32_t cur = atomicCAS(&a.table[pos], 0u, i + 1);
        if (cur == 0) {
            a.rank1[i] = count_key(a.counts, a.ht, a.bloom, t.keys[i]);
            return;
        }
        if (tuple_equal_cg(t, cur - 1, i)) {
            atomicAdd(reinterpret_cast<unsigned long long*>(&t.mult[cur - 1]), (unsigned long long)m);
            a.rank1[i] = 0;
            return;
        }
        pos = (pos + 1) & mask;
    }
    a.rank1[i] = 0;
    record_error(a.err, kErrCapacity);
}

// Writes tuple i of a build (multiplicity 0 for a NULL key or one that a
// sideways filter cannot hold: such a tuple represents nothing). A tuple of a
// distinct build represents itself and is counted into its bucket here; the
// others are folded by aggregate_tuple in a later launch, which sees every
// tuple written (no fence needed here).
__device__ __forceinline__ void emit_tuple(const BuildArgs& a, uint32_t i) {
    const uint32_t row = item_row(a.in, i);
    uint64_t kv = 0;
    bool key_ok;
    if (a.key_stage >= 0) {
        // The key is an attribute of an input probed by this pipeline.
        const HTView& src = a.ps.ht[a.key_stage];
        const uint32_t e = a.in.ents[a.key_stage][i];
        key_ok = !ht_slot_null(src, e, a.key_slot);
        if (key_ok) kv = ht_slot(src, e, a.key_slot);
    } else {
        key_ok = row < a.key.nrows && col_get(a.key, row, kv);
        if (row >= a.key.nrows) record_error(a.err, kErrRowRange);
    }
    if (key_ok && a.rbloom && !bloom_may_contain(a.rbloom, a.rlog2w, uint32_t(kv))) key_ok = false;
    const uint64_t m = key_ok ? item_mult(a.in, i) : 0ull;
    const TupleBuf& t = a.tb;
    t.keys[i] = kv;
    t.mult[i] = m;
    uint32_t nulls = 0;
    for (int j = 0; j < a.src.n; j++) {
        uint64_t v = 0;
        if (!slot_value(a.src.s[j], a.in, i, row, a.ps, v)) {
            nulls |= 1u << j;
            v = 0;
        }
        t.pay[size_t(i) * t.width + j] = v;
    }
    if (t.pnull) t.pnull[i] = nulls;
    if (m == 0)
        a.rank1[i] = 0;
    else if (a.distinct)
        a.rank1[i] = count_key(a.counts, a.ht, a.bloom, kv);
}

__global__ void __launch_bounds__(256) k_emit(BuildArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.tb.count) return;
    if (a.in.dcount && i >= *a.in.dcount) {  // beyond the items: represents nothing
        a.rank1[i] = 0;
        a.tb.mult[i] = 0;
        return;
    }
    emit_tuple(a, i);
}

__global__ void __launch_bounds__(256) k_aggregate(BuildArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.tb.count) aggregate_tuple(a, i);
}

// Places representative i as an entry of its bucket. (Its multiplicity grew by
// atomics, perhaps earlier in this launch: read through L2.)
__device__ __forceinline__ void place_tuple(const TupleBuf& t, const uint32_t* rank1, const HTView& ht, uint32_t* err,
                                            uint32_t i) {
    const uint32_t r1 = rank1[i];
    uint32_t pos;
    if (!r1 || !place_key(ht, t.keys[i], r1 - 1, err, pos)) return;
    const_cast<uint64_t*>(ht.mult)[pos] = __ldcg(t.mult + i);
    if (ht.pnull) const_cast<uint32_t*>(ht.pnull)[pos] = t.pnull[i];
    uint64_t* dst = const_cast<uint64_t*>(ht.ent) + size_t(pos) * (1 + ht.width) + 1;
    const uint64_t* src = t.pay + size_t(i) * t.width;
    for (uint32_t j = 0; j < t.width; j++) dst[j] = src[j];
}

__global__ void __launch_bounds__(256) k_place(TupleBuf t, const uint32_t* __restrict__ rank1, HTView ht,
                                               uint32_t* __restrict__ err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < t.count) place_tuple(t, rank1, ht, err, i);
}

__device__ __forceinline__ int leaf_of(const uint32_t* start, int n, uint32_t x) {
    int b = 0;
    while (b + 1 < n && x >= start[b + 1]) b++;
    return b;
}

// Exclusive prefix of v over the block (256 threads), in thread order.
__device__ __forceinline__ uint32_t block_excl_u32(uint32_t v, uint32_t& total) {
    __shared__ uint32_t ws[8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= uint32_t(o)) inc += u;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    uint32_t base = 0;
    total = 0;
    for (uint32_t w = 0; w < 8; w++) {
        if (w < warp) base += ws[w];
        total += ws[w];
    }
    return base + inc - v;
}

// Bucket ranges: a block takes a tile of 1024 buckets of one build, reserves
// the entries it counts with one atomic and writes each bucket's first entry
// and length (thread k: counts 4k .. 4k + 3; nb is a multiple of 16).
__global__ void __launch_bounds__(256) k_bucket_ranges(BucketTiles t) {
    const int b = leaf_of(t.tile_start, t.n, blockIdx.x);
    const uint32_t i0 = (blockIdx.x - t.tile_start[b]) * kBucketTile + 4 * threadIdx.x;
    const BucketTiles::Build& B = t.b[b];
    uint4 c = make_uint4(0, 0, 0, 0);
    if (i0 < B.nb) c = *reinterpret_cast<const uint4*>(B.counts + i0);
    uint32_t total;
    uint32_t run = block_excl_u32(c.x + c.y + c.z + c.w, total);
    __shared__ uint32_t base;
    if (threadIdx.x == 0) base = total ? atomicAdd(B.entries, total) : 0u;
    __syncthreads();
    if (i0 >= B.nb) return;
    run += base;
    uint4* out = B.buckets + i0;
    out[0] = make_uint4(run, c.x, 0, 0);
    out[1] = make_uint4(run + c.x, c.y, 0, 0);
    out[2] = make_uint4(run + c.x + c.y, c.z, 0, 0);
    out[3] = make_uint4(run + c.x + c.y + c.z, c.w, 0, 0);
}

// Whether a key repeats in the warp's buckets, a bucket a lane; all lanes
// together, those without a bucket with there = false. A bucket of more than
// kLaneBucket entries is the whole warp's: Zipf-repeated keys held single lanes
// for 9.7 ms; the query that has them takes 1.0 ms in all on its first run now.
// (flags: what other blocks have found, looked at along a long bucket only. A
// block sets it once, with set_repeats: a store for each of 50,000 buckets of
// repeated keys, or a look at the word by every warp, is 60 to 270 us.)
constexpr uint32_t kLaneBucket = 8;
__device__ __forceinline__ bool repeats(const HTView& ht, uint32_t first, uint32_t i) {  // entry first + i, of those before
    const uint64_t key = __ldcg(ht.ent + size_t(first + i) * (1 + ht.width));
    for (uint32_t j = 0; j < i; j += 4) {
        uint64_t q[4];
#pragma unroll
        for (int u = 0; u < 4; u++) q[u] = j + u < i ? __ldcg(ht.ent + size_t(first + j + u) * (1 + ht.width)) : ~key;
        if (q[0] == key || q[1] == key || q[2] == key || q[3] == key) return true;
    }
    return false;
}
__device__ __forceinline__ bool key_repeats(const HTView& ht, uint32_t b, bool there, const uint32_t* flags) {
    const uint32_t lane = threadIdx.x & 31;
    const uint4 k = there ? __ldcg(ht.buckets + b) : make_uint4(0, 0, 0, 0);
    bool found = false;
    if (k.y <= kLaneBucket && (k.y > 2 || (k.y == 2 && k.z == k.w)))
        for (uint32_t i = 1; i < k.y && !found; i++) found = repeats(ht, k.x, i);
    found = __any_sync(0xffffffffu, found);
    for (uint32_t left = __ballot_sync(0xffffffffu, k.y > kLaneBucket); left && !found; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const uint32_t x = __shfl_sync(0xffffffffu, k.x, src), y = __shfl_sync(0xffffffffu, k.y, src);
        // Long bucket: assume repeats (only steers capacity choices).
        found = y > 256 || (!ht.wide && __shfl_sync(0xffffffffu, k.z, src) == __shfl_sync(0xffffffffu, k.w, src));
        for (uint32_t i = lane; i - lane < y && !found; i += 32)
            found = __any_sync(0xffffffffu, (i < y && repeats(ht, x, i)) || __ldcg(flags) != 0);
    }
    return found;
}
__device__ __forceinline__ void set_repeats(bool found, uint32_t* flags) {
    if (__syncthreads_or(found) && threadIdx.x == 0) flags[0] = 1;
}
// The flag of the multiplicities, by entries (flags[2] of them, placed): with
// their buckets, one of two million entries was one warp's for 20 ms.
__device__ __forceinline__ void flag_mults(const HTView& ht, uint32_t t, uint32_t all, uint32_t* flags) {
    if (!ht.mult) return;
    const uint32_t n = min(__ldcg(flags + 2), ht.nentries);
    bool above = false;
    for (uint32_t e = t; e < n; e += all) above = above || __ldcg(ht.mult + e) > 1;
    if (above) flags[1] = 1;
}

__global__ void __launch_bounds__(256) k_ht_flags(HTView ht, uint32_t nbuckets, uint32_t* flags) {
    const uint32_t lane = threadIdx.x & 31, t = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
    flag_mults(ht, t, all, flags);
    bool found = false;
    for (uint32_t b = t; b - lane < nbuckets && !found; b += all) found = key_repeats(ht, b, b < nbuckets, flags);
    set_repeats(found, flags);
}

// Bucket ranges by a cluster: thread t of `all`, a warp a run of 32 buckets (or all
// 16), each run's entries reserved with one atomic.
__device__ __forceinline__ void cluster_ranges(const uint32_t* counts, const HTView& ht, uint32_t nb, uint32_t* entries,
                                               uint32_t t, uint32_t all) {
    uint4* buckets = const_cast<uint4*>(ht.buckets);
    const uint32_t lane = t & 31;
    for (uint32_t w = t >> 5; w * 32 < nb; w += all / 32) {
        const uint32_t b = w * 32 + lane;
        const uint32_t n = b < nb ? __ldcg(counts + b) : 0u;
        uint32_t inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += u;
        }
        uint32_t first = 0;
        if (lane == 31 && inc) first = atomicAdd(entries, inc);
        first = __shfl_sync(0xffffffffu, first, 31);
        if (b < nb) buckets[b] = make_uint4(first + inc - n, n, 0, 0);
    }
}
__device__ __forceinline__ void cluster_zero(uint32_t* p, uint32_t words, uint32_t t, uint32_t all) {  // 16-byte multiples
    for (uint32_t i = t; i < words / 4; i += all) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
}

// A small build fed by probes, whole: the passes above (zeroing, emit,
// aggregation, ranges, places, flags) in one launch, with a cluster barrier
// where they have a launch. Five launches and a memset cost the host about 20
// us a build when a query is not replayed. Bound: the passes' latencies, each
// row's chain of atomics among them, over the cluster's 8,192 threads.
constexpr int kFedCtas = 8, kFedThreads = 1024;
__global__ void __cluster_dims__(kFedCtas, 1, 1) __launch_bounds__(kFedThreads) k_fed_cluster(FedBuild f) {
    const cg::cluster_group cluster = cg::this_cluster();
    const BuildArgs& a = f.a;
    constexpr uint32_t all = kFedCtas * kFedThreads;
    const uint32_t t = blockIdx.x * kFedThreads + threadIdx.x;
    const uint32_t n = a.in.dcount ? min(a.tb.count, *a.in.dcount) : a.tb.count;
    if (!a.distinct) cluster_zero(a.table, 1u << a.tlog2, t, all);
    cluster_zero(a.counts, f.nb, t, all);
    if (a.bloom) cluster_zero(a.bloom, 1u << a.ht.bloom_log2, t, all);
    if (t < 3) f.dflags[t] = 0;
    if (a.distinct) cluster.sync();  // the emit counts
    for (uint32_t i = t; i < n; i += all) emit_tuple(a, i);
    cluster.sync();
    if (!a.distinct) {
        for (uint32_t i = t; i < n; i += all) aggregate_tuple(a, i);
        cluster.sync();
    }
    cluster_ranges(a.counts, a.ht, f.nb, f.dflags + 2, t, all);
    cluster.sync();
    for (uint32_t i = t; i < n; i += all) place_tuple(a.tb, a.rank1, a.ht, a.err, i);
    if (!f.flags) return;
    cluster.sync();
    flag_mults(a.ht, t, all, f.dflags);
    bool found = false;
    for (uint32_t b = t; b - (t & 31) < f.nb && !found; b += all) found = key_repeats(a.ht, b, b < f.nb, f.dflags);
    set_repeats(found, f.dflags);
}

// ---- leaf builds of a query, batched ----
//
// The leaves of a query build together, each pass one launch over all of
// them (blocks find their build from prefix sums of the builds' sizes).

// Row i's key when the row takes part in the build: not NULL and, under a
// sideways restriction, possibly in the restricting filter (a row whose key
// it cannot hold joins nothing).
__device__ __forceinline__ bool leaf_key(const LeafBuild& L, uint32_t i, uint64_t& kv) {
    return col_get(L.key, i, kv) && (!L.rbloom || bloom_may_contain(L.rbloom, L.rlog2w, uint32_t(kv)));
}

// Row i's entry: its key and the values of its payload columns.
__device__ __forceinline__ void leaf_place(const LeafBuild& L, uint32_t i, uint64_t kv, uint32_t rank, uint32_t* err) {
    uint32_t pos;
    if (!place_key(L.ht, kv, rank, err, pos)) return;
    uint64_t* dst = const_cast<uint64_t*>(L.ht.ent) + size_t(pos) * (1 + L.ht.width) + 1;
    uint32_t nulls = 0;
    for (int j = 0; j < L.nslots; j++) {
        uint64_t v = 0;
        if (!column_value(L.cols[j], i, v)) {
            nulls |= 1u << j;
            v = 0;
        }
        dst[j] = v;
    }
    if (L.ht.pnull) const_cast<uint32_t*>(L.ht.pnull)[pos] = nulls;
}

// Blocks of 256 rows, each within one build (block_start: prefix of the
// builds' block counts), so a block's build and its arguments are uniform.
__device__ __forceinline__ bool leaf_row(const LeafBatch& B, int& b, uint32_t& i) {
    b = leaf_of(B.block_start, B.n, blockIdx.x);
    i = (blockIdx.x - B.block_start[b]) * blockDim.x + threadIdx.x;
    return i < B.l[b].rows;
}

__global__ void __launch_bounds__(256) k_leaf_count(LeafBatch B) {
    int b;
    uint32_t i;
    if (!leaf_row(B, b, i)) return;
    const LeafBuild& L = B.l[b];
    uint64_t kv = 0;
    L.rank1[i] = leaf_key(L, i, kv) ? count_key(L.counts, L.ht, L.bloom, kv) : 0u;
}

__global__ void __launch_bounds__(256) k_leaf_place(LeafBatch B) {
    int b;
    uint32_t i;
    if (!leaf_row(B, b, i)) return;
    const LeafBuild& L = B.l[b];
    const uint32_t r1 = L.rank1[i];
    uint64_t kv = 0;
    if (r1 && col_get(L.key, i, kv)) leaf_place(L, i, kv, r1 - 1, B.err);
}

// A quarter tile a block: a thread a bucket, so the entries that buckets of two
// keys and more compare are read side by side (24 tiles, a thread four buckets
// one after another: 13 us; a thread one bucket 7 us).
__global__ void __launch_bounds__(256) k_leaf_flags(LeafBatch B) {
    const uint32_t tile = blockIdx.x / (kBucketTile / 256);
    const int b = leaf_of(B.tile_start, B.n, tile);
    const LeafBuild& L = B.l[b];
    const uint32_t i = (tile - B.tile_start[b]) * kBucketTile + (blockIdx.x % (kBucketTile / 256)) * 256 + threadIdx.x;
    set_repeats(key_repeats(L.ht, i, i < L.nb, L.dflags), L.dflags);
}

// Leaves of at most kClusterLeafRows rows: a cluster of eight CTAs builds one
// table in one launch. The passes are the ones above, over buffers in L2, with
// a cluster barrier (its CTAs are resident together) where they have a launch;
// the zeroing is a pass too, so no memset goes before.
constexpr int kClusterCtas = 8;
constexpr int kClusterThreads = 512;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads) k_leaf_cluster(LeafBatch B) {
    const cg::cluster_group cluster = cg::this_cluster();
    const LeafBuild& L = B.l[blockIdx.x / kClusterCtas];
    const uint32_t all = kClusterCtas * kClusterThreads;
    const uint32_t t = (blockIdx.x % kClusterCtas) * kClusterThreads + threadIdx.x;
    cluster_zero(L.counts, L.nb, t, all);
    if (L.bloom) cluster_zero(L.bloom, 1u << L.ht.bloom_log2, t, all);
    if (t < 3) L.dflags[t] = 0;
    cluster.sync();
    for (uint32_t i = t; i < L.rows; i += all) {
        uint64_t kv = 0;
        L.rank1[i] = leaf_key(L, i, kv) ? count_key(L.counts, L.ht, L.bloom, kv) : 0u;
    }
    cluster.sync();
    cluster_ranges(L.counts, L.ht, L.nb, L.dflags + 2, t, all);
    cluster.sync();
    for (uint32_t i = t; i < L.rows; i += all) {
        const uint32_t r1 = L.rank1[i];  // this thread's own
        uint64_t kv = 0;
        if (r1 && col_get(L.key, i, kv)) leaf_place(L, i, kv, r1 - 1, B.err);
    }
    if (!B.flags) return;
    cluster.sync();
    bool found = false;
    for (uint32_t b = t; b - (t & 31) < L.nb && !found; b += all) found = key_repeats(L.ht, b, b < L.nb, L.dflags);
    set_repeats(found, L.dflags);
}

// Hit counts of evenly spaced sample rows against every probe of a pipeline:
// blockIdx.y selects the probe.
__global__ void k_sample_probes(SampleSet set, uint32_t nsample, uint32_t* hits) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const SampleProbe& sp = set.p[blockIdx.y];
    if (i >= nsample || sp.key.nrows == 0) return;
    const uint32_t row = uint32_t((uint64_t(i) * sp.key.nrows) / nsample);
    uint64_t v;
    if (!col_get(sp.key, row, v)) return;
    bucket_matches(sp.ht, ht_bucket(sp.ht, v), v, [&](uint32_t) {
        atomicAdd(hits + blockIdx.y, 1u);
        return false;
    });
}

} // namespace

int emit_aggregate(const BuildArgs& a, cudaStream_t st) {
    if (!a.tb.count) return 0;
    const uint32_t blocks = (a.tb.count + 255) / 256;
    k_emit<<<blocks, 256, 0, st>>>(a);
    if (a.distinct) return 1;
    k_aggregate<<<blocks, 256, 0, st>>>(a);
    return 2;
}

int build_fed_cluster(const FedBuild& f, cudaStream_t st) {
    if (!f.a.tb.count) return 0;
    k_fed_cluster<<<kFedCtas, kFedThreads, 0, st>>>(f);
    return 1;
}

int place_tuples(const TupleBuf& t, const uint32_t* rank1, const uint32_t* counts, uint32_t* entries, uint32_t nb,
                 const HTView& ht, uint32_t* err, cudaStream_t st) {
    if (!t.count) return 0;
    BucketTiles tiles{};
    tiles.b[0] = {counts, const_cast<uint4*>(ht.buckets), entries, nb};
    tiles.tile_start[1] = (nb + kBucketTile - 1) / kBucketTile;
    tiles.n = 1;
    k_bucket_ranges<<<tiles.tile_start[1], 256, 0, st>>>(tiles);
    k_place<<<(t.count + 255) / 256, 256, 0, st>>>(t, rank1, ht, err);
    return 2;
}

int ht_flags(HTView ht, uint32_t nbuckets, uint32_t* flags, int num_sms, cudaStream_t st) {
    if (!ht.nentries) return 0;
    const uint32_t blocks = std::min<uint32_t>((nbuckets + 255) / 256, uint32_t(num_sms) * 8);
    k_ht_flags<<<blocks, 256, 0, st>>>(ht, nbuckets, flags);
    return 1;
}

int build_cluster_leaves(const LeafBatch& batch, cudaStream_t st) {
    if (batch.n <= 0) return 0;
    k_leaf_cluster<<<unsigned(batch.n * kClusterCtas), kClusterThreads, 0, st>>>(batch);
    return 1;
}

int build_leaves(const LeafBatch& batch, cudaStream_t st) {
    const uint32_t blocks = batch.block_start[batch.n], tiles = batch.tile_start[batch.n];
    if (batch.n <= 0 || blocks == 0) return 0;
    BucketTiles bt{};
    bt.n = batch.n;
    for (int b = 0; b < batch.n; b++) {
        const LeafBuild& L = batch.l[b];
        bt.b[b] = {L.counts, const_cast<uint4*>(L.ht.buckets), L.dflags + 2, L.nb};
        bt.tile_start[b + 1] = batch.tile_start[b + 1];
    }
    k_leaf_count<<<blocks, 256, 0, st>>>(batch);
    k_bucket_ranges<<<tiles, 256, 0, st>>>(bt);
    k_leaf_place<<<blocks, 256, 0, st>>>(batch);
    if (!batch.flags) return 3;
    k_leaf_flags<<<tiles * (kBucketTile / 256), 256, 0, st>>>(batch);
    return 4;
}

int sample_probes(const SampleSet& set, uint32_t nsample, uint32_t* hits, cudaStream_t st) {
    if (!nsample || set.n <= 0) return 0;
    k_sample_probes<<<dim3((nsample + 255) / 256, unsigned(set.n)), 256, 0, st>>>(set, nsample, hits);
    return 1;
}

} // namespace bj
