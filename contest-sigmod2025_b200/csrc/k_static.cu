// Join-count entry point that allocates nothing (bj_join_count_static).
//
// Some callers of this library cannot call cudaMalloc: their device memory is
// owned by another allocator (a framework's caching pool, or a fixed budget
// carved out at start-up), or they issue work from code where cudaMalloc's
// implicit device synchronisation is not acceptable. For them this entry point
// counts the rows of a two-table INT32 equi-join -- the row count bj_execute
// returns for Scan(A) JOIN Scan(B) on those columns -- using only the buffers
// the caller passes and one fixed scratch array compiled into the library.
//
// The scratch is a file-scope __device__ array of kStaticSlots 64-bit slots
// (4 MiB); every GPU that loads the library holds it until the process exits.
// Host code must not take its address directly (the host-side name is a
// stand-in, not a device address): the device address is obtained once per
// device with cudaGetSymbolAddress, with that device current, on the first
// call made on it. Make that first call before any stream capture.
//
// All calls share the array, and it keeps the last call's contents; each call
// clears it before use. Calls that overlap on the GPU (e.g. on two streams at
// once) race on the array and give wrong counts: serialise them.
//
// Bad input is reported through the count: a page whose header cannot be an
// INT32 page, or build pages holding more non-null values than build_rows,
// set a flag word in the scratch, and the last kernel then writes ~0ull
// (UINT64_MAX) to *out_count. The call itself only enqueues work, so its
// return status cannot carry what the kernels find.
//
// The device address is cached per device for the life of the process; after
// cudaDeviceReset the module may load at another address, so the entry point
// must not be used across a device reset.
#include "../../include/b200join.h"
#include "device.cuh"

#include <cuda_runtime.h>

#include <mutex>

namespace bj {
namespace {

constexpr uint32_t kStaticLog2 = 19;
constexpr uint32_t kStaticSlots = 1u << kStaticLog2;     // 4 MiB of 64-bit slots (+256 B)
constexpr uint64_t kStaticMaxBuildRows = kStaticSlots / 2; // load factor <= 1/2
constexpr uint64_t kSlotEmpty = ~0ull;

// Slot: key in the high 32 bits, count of build rows with that key in the low
// 32 bits. The all-ones pattern cannot occur as a filled slot because a count
// never reaches 2^32 - 1 (at most kStaticMaxBuildRows), so a key of -1
// (0xFFFFFFFF) is stored like any other. A call uses the first 2^log2 slots, at
// least twice build_rows: a small build clears and probes a table that stays in
// L1. The word after all slots counts the values pages brought, so pages
// holding more values than the caller said can never fill the table past one
// half; the words after that collect error bits and the probe blocks done.
constexpr uint32_t kCounterWord = kStaticSlots;
constexpr uint32_t kErrorWord = kStaticSlots + 1;
constexpr uint32_t kDoneWord = kStaticSlots + 2;
constexpr unsigned long long kErrBadPage = 1;     // a page header that cannot be an INT32 page
constexpr unsigned long long kErrTooManyRows = 2; // more non-null build values than build_rows
static __device__ __align__(256) unsigned long long g_join_scratch[kStaticSlots + 32];

constexpr int kPerThread = 8;                       // values a thread has in flight
constexpr uint32_t kPageSpan = 256 * kPerThread;    // more than the values of any page

__global__ void __launch_bounds__(256) k_static_clear(unsigned long long* slots, uint32_t n, unsigned long long* out_count) {
    for (uint32_t i = 2 * (blockIdx.x * blockDim.x + threadIdx.x); i < n; i += 2 * gridDim.x * blockDim.x)
        *reinterpret_cast<ulonglong2*>(slots + i) = make_ulonglong2(kSlotEmpty, kSlotEmpty);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        slots[kCounterWord] = 0;
        slots[kErrorWord] = 0;
        slots[kDoneWord] = 0;
        *out_count = 0;
    }
}

// Non-null INT32 values of page p (stored densely, so the bitmap need not be
// read: a join count needs only the multiset of keys), or 0, flagged, for a
// page that cannot be an INT32 page.
__device__ __forceinline__ uint32_t page_values(const uint8_t* pg, unsigned long long* slots) {
    const uint32_t hdr = *reinterpret_cast<const uint32_t*>(pg), n = hdr & 0xffff, nn = hdr >> 16;
    if (nn <= n && 4 + 4 * nn + ((n + 7) >> 3) <= kPageSize) return nn;
    if (threadIdx.x == 0) atomicOr(&slots[kErrorWord], kErrBadPage);
    return 0;
}

// A quarter page a block: its 512 values are reserved with one atomic, two a
// thread inserted.
constexpr uint32_t kBuildParts = 4, kBuildSpan = kPageSpan / kBuildParts;
__global__ void __launch_bounds__(256) k_static_build(const uint8_t* pages, uint64_t npages, uint64_t build_rows,
                                                      unsigned long long* slots, uint32_t log2) {
    __shared__ int fits;
    const uint32_t mask = (1u << log2) - 1;
    for (uint64_t u = blockIdx.x; u < npages * kBuildParts; u += gridDim.x) {
        const uint8_t* pg = pages + (u / kBuildParts) * kPageSize;
        const uint32_t first = uint32_t(u % kBuildParts) * kBuildSpan;
        const uint32_t end = min(page_values(pg, slots), first + kBuildSpan);
        if (first >= end) continue;  // block-uniform
        if (threadIdx.x == 0) {
            fits = atomicAdd(&slots[kCounterWord], (unsigned long long)(end - first)) + (end - first) <= build_rows;
            if (!fits) atomicOr(&slots[kErrorWord], kErrTooManyRows);
        }
        __syncthreads();
        const bool take = fits;
        __syncthreads();
        if (!take) continue;
        for (uint32_t i = first + threadIdx.x; i < end; i += 256) {
            const uint32_t key = reinterpret_cast<const uint32_t*>(pg + 4)[i];
            uint32_t pos = uint32_t(key_hash(key) >> (64 - log2));
            // At most build_rows values are inserted: the table stays at most half full.
            for (uint32_t step = 0; step <= mask; step++) {
                unsigned long long cur = slots[pos];
                if (cur == kSlotEmpty) {
                    cur = atomicCAS(&slots[pos], kSlotEmpty, (static_cast<unsigned long long>(key) << 32) | 1ull);
                    if (cur == kSlotEmpty) break;
                }
                if (uint32_t(cur >> 32) == key) {
                    atomicAdd(&slots[pos], 1ull);
                    break;
                }
                pos = (pos + 1) & mask;
            }
        }
    }
}

// A page a block at a time, kPerThread values a thread, their first slots in
// flight together. The last block to finish replaces the count by ~0ull when
// an error was flagged. No more blocks than are resident together: a block's end
// is two atomics and a fence (16M rows against 500 keys 64.7 us with a block a
// page, 54.6 so; against 5,000 87 and 54).
constexpr uint64_t kProbeBlocks = 148 * 6;
__global__ void __launch_bounds__(256, 6) k_static_probe(const uint8_t* pages, uint64_t npages, unsigned long long* slots,
                                                      uint32_t log2, unsigned long long* out_count) {
    const uint32_t mask = (1u << log2) - 1;
    unsigned long long mine = 0;
    for (uint64_t p = blockIdx.x; p < npages; p += gridDim.x) {
        const uint8_t* pg = pages + p * kPageSize;
        const uint32_t nn = page_values(pg, slots);
        uint32_t key[kPerThread];
        unsigned long long cur[kPerThread];
#pragma unroll
        for (int k = 0; k < kPerThread; k++) {
            const uint32_t i = threadIdx.x + 256 * k;
            key[k] = i < nn ? __ldg(reinterpret_cast<const uint32_t*>(pg + 4) + i) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kPerThread; k++)
            cur[k] = threadIdx.x + 256 * k < nn ? __ldg(slots + uint32_t(key_hash(key[k]) >> (64 - log2))) : kSlotEmpty;
#pragma unroll
        for (int k = 0; k < kPerThread; k++) {
            uint32_t pos = uint32_t(key_hash(key[k]) >> (64 - log2));
            for (uint32_t step = 0; step <= mask && cur[k] != kSlotEmpty; step++) {
                if (uint32_t(cur[k] >> 32) == key[k]) {
                    mine += cur[k] & 0xffffffffull;
                    break;
                }
                pos = (pos + 1) & mask;
                cur[k] = __ldg(slots + pos);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    __shared__ unsigned long long part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mine;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; w++) mine += part[w];
    if (mine) atomicAdd(out_count, mine);
    __threadfence();
    if (atomicAdd(&slots[kDoneWord], 1ull) + 1 == gridDim.x && atomicOr(&slots[kErrorWord], 0ull) != 0)
        atomicExch(out_count, ~0ull);
}

// The same last step for a call without probe pages.
__global__ void k_static_finish(const unsigned long long* slots, unsigned long long* out_count) {
    if (slots[kErrorWord] != 0) *out_count = ~0ull;
}

// Device address of g_join_scratch, resolved once per device.
std::mutex g_static_mu;
unsigned long long* g_static_ptr[64] = {};

} // namespace
} // namespace bj

extern "C" BJ_API int bj_join_count_static(const void* build_pages, uint64_t build_num_pages, uint64_t build_rows,
                                           const void* probe_pages, uint64_t probe_num_pages,
                                           unsigned long long* out_count, void* stream) {
    using namespace bj;
    if (!out_count || (build_num_pages && !build_pages) || (probe_num_pages && !probe_pages)) return BJ_ERR_INVALID;
    if (build_rows > kStaticMaxBuildRows) return BJ_ERR_INVALID;  // beyond the fixed scratch
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BJ_ERR_CUDA;
    unsigned long long* slots;
    {
        std::lock_guard<std::mutex> g(g_static_mu);
        if (!g_static_ptr[dev]) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_join_scratch) != cudaSuccess || !p) return BJ_ERR_CUDA;
            g_static_ptr[dev] = static_cast<unsigned long long*>(p);
        }
        slots = g_static_ptr[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint32_t log2 = 10;
    while ((uint64_t(1) << log2) < 2 * build_rows) log2++;
    const auto grid = [](uint64_t blocks) { return unsigned(blocks < 148 * 8 ? blocks : 148 * 8); };
    k_static_clear<<<grid((uint64_t(1) << log2) / 512), 256, 0, st>>>(slots, 1u << log2, out_count);
    if (build_num_pages)
        k_static_build<<<grid(build_num_pages * kBuildParts), 256, 0, st>>>(
            static_cast<const uint8_t*>(build_pages), build_num_pages, build_rows, slots, log2);
    if (probe_num_pages)  // probe pages are read (and checked) even when the build side is empty
        k_static_probe<<<unsigned(probe_num_pages < kProbeBlocks ? probe_num_pages : kProbeBlocks), 256, 0, st>>>(
            static_cast<const uint8_t*>(probe_pages), probe_num_pages, slots, log2, out_count);
    else
        k_static_finish<<<1, 1, 0, st>>>(slots, out_count);
    return cudaGetLastError() == cudaSuccess ? BJ_OK : BJ_ERR_CUDA;
}
