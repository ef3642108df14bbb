// The way of the estimator's feature rows from host memory to a device.
#pragma once

#include "engine.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace bj {

// n floats to BF16, to nearest even (NaN kept quiet); runs as wide as the host's
// vectors.
#if defined(__x86_64__) && defined(__GNUC__) && !defined(__clang__)
__attribute__((target_clones("avx512f", "avx2", "default")))
#endif
static void to_bf16_n(const float* in, uint16_t* out, size_t n) {
    for (size_t i = 0; i < n; i++) {
        uint32_t u;
        std::memcpy(&u, in + i, 4);
        const uint32_t r = (u + 0x7fffu + ((u >> 16) & 1u)) >> 16, nan = (u >> 16) | 0x40u;
        out[i] = uint16_t((u & 0x7fffffffu) > 0x7f800000u ? nan : r);
    }
}

// Shared by a device's estimators and freed with the last of them: a small
// pinned ring (pinning costs a millisecond or more a MB), the events of its
// places' copies and the threads that convert into it.
class RowStage {
    public:
    static std::shared_ptr<RowStage> of(int device) {
        static std::mutex m;
        static std::vector<std::weak_ptr<RowStage>> stages;
        std::lock_guard<std::mutex> g(m);
        if (stages.size() <= size_t(device)) stages.resize(size_t(device) + 1);
        std::shared_ptr<RowStage> s = stages[size_t(device)].lock();
        if (!s) stages[size_t(device)] = s = std::make_shared<RowStage>(device);
        return s;
    }

    explicit RowStage(int device)
        : device_(device), pool_(std::min(std::max(1u, std::thread::hardware_concurrency()), 8u) - 1) {
        void* p = nullptr;
        BJ_CK(cudaHostAlloc(&p, sizeof(uint16_t) * kPlaces * kPlaceWords, cudaHostAllocDefault));
        ring_ = static_cast<uint16_t*>(p);
        for (Place& l : place_)
            if (cudaEventCreateWithFlags(&l.copied, cudaEventDisableTiming) != cudaSuccess) {
                free_all();
                throw Fail{BJ_ERR_CUDA, "event creation failed"};
            }
    }
    ~RowStage() {
        for (Place& l : place_) cudaEventSynchronize(l.copied);
        free_all();
    }

    // Brings n rows to dst on `stream`: the pool's threads, or the caller alone,
    // convert parts of kPartRows rows into places of the ring and start their
    // copies. Bound: the host reading its FP32 rows. A whole prediction of 6,000
    // rows on a 16-core B200 host: 1.5 ms, where one thread converting every row
    // into pageable memory before their copy made it 8.4 ms.
    void upload(const float* f, uint64_t n, uint16_t* dst, cudaStream_t stream) {
        std::atomic<int> failed{cudaSuccess};
        const auto part = [&](size_t i) {
            const uint64_t r0 = i * kPartRows;
            const cudaError_t e = bring(f + r0 * kCols, std::min(kPartRows, n - r0), dst + r0 * kCols, stream);
            if (e != cudaSuccess) failed = e;
        };
        const size_t parts = size_t((n + kPartRows - 1) / kPartRows);
        // One upload at a time has the pool. A short one does not wait for it: 16
        // threads, each predicting with an estimator of its own, take 0.22 ms for
        // 32 rows each (0.49 where each waited its turn), 0.82 for 256 (1.3). From
        // 512 on the pool's turn is as soon: 1.9 either way.
        std::unique_lock<std::mutex> pool(m_, std::defer_lock);
        if (parts > kShortParts ? (pool.lock(), true) : parts > 1 && pool.try_lock())
            pool_.parallel_for(parts, part);
        else
            for (size_t i = 0; i < parts; i++) part(i);
        BJ_CK(cudaError_t(failed.load()));
    }

    static constexpr uint64_t kPartRows = 64;
    static constexpr size_t kCols = BJ_EST_FEATURES, kPlaces = 8, kPlaceWords = kPartRows * kCols, kShortParts = 4;

    private:
    // A place of the ring: the event of its last copy, and how many parts have
    // had it (their copies are enqueued).
    struct Place {
        cudaEvent_t copied = nullptr;
        std::atomic<uint64_t> parts{0};
    };
    cudaError_t bring(const float* f, uint64_t rows, uint16_t* dst, cudaStream_t stream) {
        // Parts take the places in turn; the part that has this one before is in
        // the hands of a running thread.
        const uint64_t turn = next_.fetch_add(1, std::memory_order_relaxed);
        Place& l = place_[turn % kPlaces];
        while (l.parts.load(std::memory_order_acquire) < turn / kPlaces) std::this_thread::yield();
        cudaError_t e = cudaSetDevice(device_);
        if (e == cudaSuccess) e = cudaEventSynchronize(l.copied);
        if (e == cudaSuccess) {
            uint16_t* to = ring_ + turn % kPlaces * kPlaceWords;
            to_bf16_n(f, to, rows * kCols);
            e = cudaMemcpyAsync(dst, to, sizeof(uint16_t) * rows * kCols, cudaMemcpyHostToDevice, stream);
            if (e == cudaSuccess) e = cudaEventRecord(l.copied, stream);
        }
        l.parts.store(turn / kPlaces + 1, std::memory_order_release);
        return e;
    }
    void free_all() {
        for (Place& l : place_)
            if (l.copied) cudaEventDestroy(l.copied);
        cudaFreeHost(ring_);
    }
    int device_;
    std::mutex m_;  // the pool's
    std::atomic<uint64_t> next_{0};
    uint16_t* ring_ = nullptr;
    Place place_[kPlaces];
    ThreadPool pool_;
};

} // namespace bj
