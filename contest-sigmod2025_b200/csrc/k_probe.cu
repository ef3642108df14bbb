// Pipeline kernels: probe stages, build-side tuple emit, output emit.
//
// Replaces the fused push pipeline of the reference
// (engine/pipeline/JoinPipeline.hpp:46-203: scan -> probe_0 -> probe_1 ->
// target, multiplicity = product of the matched tuples' multiplicities,
// :111-131) with stage kernels over item lists. An item is a row of the
// scanned input plus the hash-table entry matched by every probe so far.
// Against a table with unique keys a stage makes at most one item per input
// item, so it runs once, appending with warp-aggregated atomics and reading
// its input count on the device (no host round trip between stages).
// Otherwise it runs twice: once counting the matches, which sizes the items'
// buffers, once appending them. A query captured into a graph knows the count
// from its recording and runs the second alone.
//
// The probe itself follows HashtableProbe::operator() (engine/op/Hashtable.hpp:
// 228-241): hash the 32-bit key, find its bucket, compare every key in the
// bucket. Buckets here are contiguous runs of entries (CSR), not chains.
// INT64 keys (no reference counterpart: the reference reads every join key as
// 32 bits) hash all 64 bits and compare both halves.
#include "launch.h"

#include <algorithm>

namespace bj {
namespace {


// Entries of `ht` whose key equals `key`: calls fn(entry) for each, until it
// returns false. `key` is a value slot: an INT32 key zero-extended, or an
// INT64 key (the table is then wide and carries no bloom filter).
template <typename Fn>
__device__ __forceinline__ void for_matches(const HTView& ht, uint64_t key, bool use_bloom, Fn&& fn) {
    if (use_bloom && ht.bloom && !bloom_may_contain(ht.bloom, ht.bloom_log2, uint32_t(key))) return;
    bucket_matches(ht, ht_bucket(ht, key), key, fn);
}

// Key of item i (row `row`) for a stage: a column of the scanned input, or an
// earlier stage's payload.
__device__ __forceinline__ bool stage_key(const DevColumn& key, const KeySource& src, const Items& in, uint32_t i,
                                          uint32_t row, uint32_t* err, uint64_t& v) {
    if (src.stage >= 0) return payload_key(src, in.ents, i, v);
    if (row >= key.nrows) {
        record_error(err, kErrRowRange);
        return false;
    }
    return col_get(key, row, v);
}

// Probe stage against a table whose keys may repeat: any number of matches per
// item. A block takes `span` items: kStageItems, kPer a thread, whose buckets
// load together, or fewer where each has many matches; a lane then finds all
// matches of an item as one bit mask.
constexpr int kPer = 2;
constexpr uint32_t kStageItems = 256 * kPer;
constexpr uint32_t kStageMatches = 4096;  // matches of a block collected in shared memory

struct StageItems {
    uint64_t key[kPer];
    uint4 bucket[kPer];  // empty for an item without a key
    // Item k of lane l of this warp is number 256 k + first + l stride of the
    // block: fewer than a block's threads are dealt to its warps in turn.
    uint32_t first, stride;
    __device__ __forceinline__ uint32_t number(int k, uint32_t lane) const { return 256 * k + first + lane * stride; }
};
__device__ __forceinline__ void load_stage(StageItems& it, const Items& in, uint32_t span, const DevColumn& key,
                                           const HTView& ht, int use_bloom, const KeySource& src, uint32_t* err) {
    bool ok[kPer];
    const uint32_t warp = threadIdx.x >> 5;
    it.first = span == kStageItems ? 32 * warp : warp;
    it.stride = span == kStageItems ? 1 : 8;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const uint32_t local = it.number(k, threadIdx.x & 31), i = blockIdx.x * span + local;
        it.key[k] = 0;
        ok[k] = local < span && i < in.count && stage_key(key, src, in, i, item_row(in, i), err, it.key[k]);
    }
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        it.bucket[k] = make_uint4(0, 0, 0, 0);
        if (ok[k] && (!use_bloom || !ht.bloom || bloom_may_contain(ht.bloom, ht.bloom_log2, uint32_t(it.key[k]))))
            it.bucket[k] = ht_bucket(ht, it.key[k]);
    }
}
// Which of a bucket's first 32 entries have the key (bit j: entry j). The
// bucket holds the low halves of the first two; the keys of the others load
// four at a time.
__device__ __forceinline__ uint32_t match_mask(const HTView& ht, const uint4& b, uint64_t key) {
    const uint32_t n = min(b.y, 32u), lo = uint32_t(key);
    uint32_t m = (n >= 1 && b.z == lo ? 1u : 0u) | (n >= 2 && b.w == lo ? 2u : 0u);
    if (ht.wide) {
        const uint64_t k0 = m & 1 ? ht_key(ht, b.x) : key, k1 = m & 2 ? ht_key(ht, b.x + 1) : key;
        if (k0 != key) m &= ~1u;
        if (k1 != key) m &= ~2u;
    }
    for (uint32_t j = 2; j < n; j += 4) {
        uint64_t q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = j + i < n ? ht_key(ht, b.x + j + i) : ~key;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (q[i] == key) m |= 1u << (j + i);
    }
    return m;
}

// The entries from the 33rd of the warp's long buckets, 32 lanes on a bucket:
// a key that repeats thousands of times would otherwise hold its lane, and the
// warp, for as many dependent steps. Lanes with the same key share a walk (a key
// that repeats in the build often does in the probe): fn(group, e, hit) is
// called by all lanes together for the items of the lanes in group: entry e +
// 32 u matches when bit u of the caller's hit is set. The stages of a schema20
// query with Zipf-repeated keys: 8.0 ms with the buckets of a warp walked in
// step, 2.7 ms with each lane walking its own, 0.25 ms now. 116M items that find
// a long bucket of other keys: 235 ms with a walk an item, 8 ms.
// Entries a lane has in flight, at five blocks an SM: a replayed query that walks
// much 7.3 ms with 2, 4.4 with 4 (which spill at six blocks' 40 registers).
constexpr int kLongStep = 4;
template <typename Fn>
__device__ __forceinline__ void long_buckets(const HTView& ht, const uint4& b, uint64_t key, Fn&& fn) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t left = __ballot_sync(0xffffffffu, b.y > 32); left;) {
        const int src = __ffs(left) - 1;
        const uint32_t x = __shfl_sync(0xffffffffu, b.x, src), y = __shfl_sync(0xffffffffu, b.y, src);
        const uint64_t k = __shfl_sync(0xffffffffu, key, src);
        const uint32_t group = __ballot_sync(0xffffffffu, b.y > 32 && key == k);
        left &= ~group;
        for (uint32_t j0 = 32; j0 < y; j0 += 32 * kLongStep) {
            uint64_t q[kLongStep];
#pragma unroll
            for (int u = 0; u < kLongStep; u++) {
                const uint32_t j = j0 + 32 * u + lane;
                q[u] = j < y ? ht_key(ht, x + j) : ~k;
            }
            uint32_t hit = 0;
#pragma unroll
            for (int u = 0; u < kLongStep; u++)
                if (q[u] == k) hit |= 1u << u;
            fn(group, x + j0 + lane, hit);
        }
    }
}

// Counts the matches: *total (zero before) += them, in 64 bits.
__global__ void __launch_bounds__(256, 5) k_stage_count(Items in, DevColumn key, HTView ht, int use_bloom, KeySource src,
                                                     unsigned long long* total, uint32_t* err) {
    StageItems it;
    load_stage(it, in, kStageItems, key, ht, use_bloom, src, err);
    unsigned long long mine = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        mine += __popc(match_mask(ht, it.bucket[k], it.key[k]));
        long_buckets(ht, it.bucket[k], it.key[k],
                     [&](uint32_t group, uint32_t, uint32_t hit) { mine += __popc(hit) * __popc(group); });
    }
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    __shared__ unsigned long long part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) mine += part[w];
        if (mine) atomicAdd(total, mine);
    }
}

// Calls fn(position, item of the block, entry) for the block's matches, numbered from 0 in no
// particular order by the shared counter (zero before).
template <typename Fn>
__device__ __forceinline__ void walk_stage(const StageItems& it, const HTView& ht, uint32_t* counter, Fn&& fn) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        uint32_t m = match_mask(ht, it.bucket[k], it.key[k]);
        const uint32_t cnt = __popc(m);
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += u;
        }
        uint32_t o = 0;
        if (lane == 31 && inc) o = atomicAdd(counter, inc);
        o = __shfl_sync(0xffffffffu, o, 31) + inc - cnt;
        for (; m; m &= m - 1) fn(o++, it.number(k, lane), it.bucket[k].x + __ffs(m) - 1);
        long_buckets(ht, it.bucket[k], it.key[k], [&](uint32_t group, uint32_t e, uint32_t hit) {
            uint32_t m[kLongStep], all = 0;
#pragma unroll
            for (int u = 0; u < kLongStep; u++) {
                m[u] = __ballot_sync(0xffffffffu, (hit >> u) & 1);
                all += __popc(m[u]);
            }
            if (!all) return;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(counter, all * __popc(group));
            at = __shfl_sync(0xffffffffu, at, 0);
            for (; group; group &= group - 1) {
                const uint32_t item = it.number(k, __ffs(group) - 1);
#pragma unroll
                for (int u = 0; u < kLongStep; u++) {
                    if ((hit >> u) & 1) fn(at + __popc(m[u] & ((1u << lane) - 1)), item, e + 32 * u);
                    at += __popc(m[u]);
                }
            }
        });
    }
}

// Appends an item per match at *cursor: the block's matches collect in shared
// memory, leave together (one global atomic) and are written coalesced.
// Bound: the random sectors of buckets and keys in L2 (118 G a second). 2M rows
// against 300K entries of 100K INT64 keys, 4.2M matches, on a B200: 56 us; the
// two passes over tiles, each lane walking its bucket and writing its own matches, took
// 128 us (82 of them the second), lanes walking in step with one shared
// atomic a step 91 us. Five blocks an SM: at six, 40 registers spill what the
// walks share, and the whole query takes 154 us replayed, not 131.
__global__ void __launch_bounds__(256, 5) k_stage_emit(Items in, uint32_t span, DevColumn key, HTView ht, int use_bloom,
                                                       KeySource src, ItemsOut out, uint32_t* cursor, uint32_t capacity,
                                                       uint32_t* err) {
    __shared__ uint2 found[kStageMatches];  // (item of the block, entry)
    __shared__ uint32_t count, base;
    if (threadIdx.x == 0) count = 0;
    StageItems it;
    load_stage(it, in, span, key, ht, use_bloom, src, err);
    __syncthreads();
    walk_stage(it, ht, &count, [&](uint32_t o, uint32_t local, uint32_t e) {
        if (o < kStageMatches) found[o] = make_uint2(local, e);
    });
    __syncthreads();
    const uint32_t n = count;
    if (!n) return;
    if (threadIdx.x == 0) base = atomicAdd(cursor, n);
    __syncthreads();
    const uint32_t b = base;
    if (b + n > capacity || b + n < n) {
        if (threadIdx.x == 0) record_error(err, kErrCapacity);
        return;
    }
    auto write = [&](uint32_t o, uint32_t local, uint32_t e) {
        const uint32_t i = blockIdx.x * span + local;
        out.rows[o] = item_row(in, i);
        for (int p = 0; p < in.nprobes; p++) out.ents[p][o] = in.ents[p][i];
        out.ents[in.nprobes][o] = e;
        if (out.mult) out.mult[o] = item_mult(in, i) * ht_mult(ht, e);
    };
    if (n <= kStageMatches) {
        for (uint32_t j = threadIdx.x; j < n; j += 256) write(b + j, found[j].x, found[j].y);
        return;
    }
    // More than shared memory holds: a second walk writes them in place.
    __syncthreads();
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    walk_stage(it, ht, &count, [&](uint32_t o, uint32_t local, uint32_t e) { write(b + o, local, e); });
}

// A chain of consecutive probe stages against tables with unique keys: every
// item probes stage 0, and while it matches, the next stage, so a row that
// misses is dropped at its first miss (the fused probe_0 -> probe_1 -> ...
// of JoinPipeline.hpp:111-131, with early exit). Persistent grid-stride
// loop, at most one match per stage, warp-aggregated reservation of output
// slots.
__global__ void __launch_bounds__(256) k_probe_chain(Items in, ProbeChain ch, ItemsOut out, uint32_t* cursor,
                                                     uint32_t capacity, uint32_t* err, const uint32_t* dfirst,
                                                     uint32_t* dend) {
    const uint32_t n = in.dcount ? *in.dcount : in.count;
    const uint32_t first = dfirst ? *dfirst : 0u;
    if (dend && blockIdx.x == 0 && threadIdx.x == 0) *dend = n;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31;
    // Whole warps iterate together so the ballot sees every lane.
    for (uint32_t base = first + (blockIdx.x * blockDim.x + threadIdx.x) - lane; base < n; base += stride) {
        const uint32_t i = base + lane;
        bool hit = i < n;
        uint32_t row = 0;
        uint32_t e[kMaxChain];
        if (hit) row = item_row(in, i);
#pragma unroll
        for (int t = 0; t < kMaxChain; t++) {
            e[t] = 0;
            if (t >= ch.n || !hit) continue;
            const ChainStage& c = ch.st[t];
            uint64_t v;
            if (!stage_key(c.key, c.src, in, i, row, err, v)) {
                hit = false;
            } else {
                bool found = false;
                for_matches(c.ht, v, c.use_bloom != 0, [&](uint32_t j) {
                    e[t] = j;
                    found = true;
                    return false;  // unique keys: no other match
                });
                hit = found;
            }
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, hit);
        if (!mask) continue;
        uint32_t wbase = 0;
        if (lane == 0) wbase = atomicAdd(cursor, __popc(mask));
        wbase = __shfl_sync(0xffffffffu, wbase, 0);
        if (!hit) continue;
        const uint32_t o = wbase + __popc(mask & ((1u << lane) - 1));
        if (o >= capacity) {
            record_error(err, kErrCapacity);
            continue;
        }
        out.rows[o] = row;
        for (int p = 0; p < in.nprobes; p++) out.ents[p][o] = in.ents[p][i];
        uint64_t m = item_mult(in, i);
#pragma unroll
        for (int t = 0; t < kMaxChain; t++) {
            if (t >= ch.n) continue;
            out.ents[in.nprobes + t][o] = e[t];
            m *= ht_mult(ch.st[t].ht, e[t]);
        }
        if (out.mult) out.mult[o] = m;
    }
}

__global__ void k_items_mult(Items in, uint64_t* mult_out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < in.count) mult_out[i] = item_mult(in, i);
}

__global__ void __launch_bounds__(256) k_emit_output(Items in, const uint64_t* out_off, SlotSources src, ProbeSet ps,
                                                     FlatOut out, uint32_t* err) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= in.count) return;
    uint32_t row = item_row(in, i);
    // Without offsets every item is one output row.
    uint64_t o0 = out_off ? out_off[i] : i, o1 = out_off ? out_off[i + 1] : i + 1;
    for (int j = 0; j < src.n; j++) {
        if (!out.vals[j]) continue;  // a slot the page writer reads from the items
        uint64_t v = 0;
        bool ok = slot_value(src.s[j], in, i, row, ps, v);
        for (uint64_t o = o0; o < o1; o++) {
            out.vals[j][o] = ok ? v : 0;
            out.valid[j][o] = ok;
        }
    }
}

} // namespace

int probe_stage_count(const Items& in, const DevColumn& key, const HTView& ht, bool use_bloom, const KeySource& src,
                      unsigned long long* total, uint32_t* err, cudaStream_t st) {
    if (!in.count) return 0;
    k_stage_count<<<(in.count - 1) / kStageItems + 1, 256, 0, st>>>(in, key, ht, use_bloom, src, total, err);
    return 1;
}

int probe_stage(const Items& in, const DevColumn& key, const HTView& ht, bool use_bloom, const KeySource& src,
                const ItemsOut& out, uint32_t* cursor, uint32_t capacity, uint32_t* err, cudaStream_t st) {
    if (!in.count) return 0;
    // `capacity` is the matches there are. A block whose items have more than it
    // collects walks their buckets twice, and a few hundred items with thousands
    // each would be one block's: fewer items a block then (2,000 items with 1,000
    // matches each: the query 1.15 ms with 512 a block, 0.11 with 8).
    uint32_t span = kStageItems;
    while (span > 8 && uint64_t(span) * capacity > uint64_t(in.count) * (kStageMatches / 2)) span /= 2;
    k_stage_emit<<<(in.count - 1) / span + 1, 256, 0, st>>>(in, span, key, ht, use_bloom, src, out, cursor, capacity,
                                                            err);
    return 1;
}

int probe_chain_unique(const Items& in, const ProbeChain& chain, ItemsOut out, uint32_t* cursor, uint32_t capacity,
                       uint32_t* err, int num_sms, cudaStream_t st, const uint32_t* dfirst, uint32_t* dend) {
    if (!in.count || chain.n <= 0) return 0;
    uint32_t blocks = std::min<uint32_t>((in.count + 255) / 256, uint32_t(num_sms) * 8);
    k_probe_chain<<<blocks, 256, 0, st>>>(in, chain, out, cursor, capacity, err, dfirst, dend);
    return 1;
}

int items_mult(const Items& in, uint64_t* mult_out, cudaStream_t st) {
    if (!in.count) return 0;
    k_items_mult<<<(in.count + 255) / 256, 256, 0, st>>>(in, mult_out);
    return 1;
}

int emit_output(const Items& in, const uint64_t* out_off, const SlotSources& src, const HTView* probes, FlatOut out,
                uint32_t* err, cudaStream_t st) {
    if (!in.count) return 0;
    k_emit_output<<<(in.count + 255) / 256, 256, 0, st>>>(in, out_off, src, make_probe_set(probes, in.nprobes), out,
                                                          err);
    return 1;
}

} // namespace bj
