// RowStage (csrc/row_stage.h) on a CUDA runtime of the test's own, whose copies run later, in order, on a thread: uploads
// of many threads at once arrive whole, and a short one does not wait for a long one to be converted.
#include "row_stage.h"

#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <random>

static std::mutex g_m;
static std::condition_variable g_cv;
struct Copy {
    void* dst;
    const void* src;
    size_t bytes;
};
static std::deque<Copy> g_copies;
static uint64_t g_enqueued = 0, g_done = 0;
static bool g_stop = false;
static void* g_held = nullptr;  // a copy to here is not enqueued while it is set
static bool g_holding = false;
static cudaError_t g_answer = cudaSuccess;

static void copy_engine() {
    std::unique_lock<std::mutex> g(g_m);
    for (;;) {
        g_cv.wait(g, [] { return g_stop || !g_copies.empty(); });
        if (g_copies.empty()) return;
        const Copy c = g_copies.front();
        g_copies.pop_front();
        g.unlock();
        if ((g_done & 3) == 0) std::this_thread::yield();
        std::memcpy(c.dst, c.src, c.bytes);
        g.lock();
        g_done++;
        g_cv.notify_all();
    }
}

extern "C" {
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    std::unique_lock<std::mutex> g(g_m);
    if (g_answer != cudaSuccess) return g_answer;
    if (dst == g_held) {
        g_holding = true;
        g_cv.notify_all();
        g_cv.wait(g, [&] { return dst != g_held; });
    }
    g_copies.push_back({dst, src, bytes});
    g_enqueued++;
    g_cv.notify_all();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(new uint64_t(0));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete reinterpret_cast<uint64_t*>(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::mutex> g(g_m);
    *reinterpret_cast<uint64_t*>(e) = g_enqueued;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::unique_lock<std::mutex> g(g_m);
    const uint64_t upto = *reinterpret_cast<uint64_t*>(e);
    g_cv.wait(g, [&] { return g_done >= upto; });
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
}

using bj::RowStage;
constexpr size_t kCols = RowStage::kCols;

static uint16_t bf16_of(float f) {  // f is a small whole number: its upper half
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return uint16_t(u >> 16);
}

struct Rows {
    std::vector<float> f;
    std::vector<uint16_t> got;
    uint64_t n;
    Rows(uint64_t rows, unsigned seed) : f(rows * kCols), got(rows * kCols, 0xffff), n(rows) {
        std::mt19937 rng(seed);
        for (float& x : f) x = float(int(rng() % 200) - 100);
    }
    bool arrived() const {
        for (size_t i = 0; i < f.size(); i++)
            if (got[i] != bf16_of(f[i])) return false;
        return true;
    }
};
static void drain() {
    std::unique_lock<std::mutex> g(g_m);
    g_cv.wait(g, [] { return g_done == g_enqueued; });
}

#define CHECK(x)                                                  \
    if (!(x)) {                                                   \
        std::printf("line %d: %s does not hold\n", __LINE__, #x); \
        std::fflush(stdout);                                      \
        std::_Exit(1);                                            \
    }

int main() {
    std::thread engine(copy_engine);
    {
        const std::shared_ptr<RowStage> stage = RowStage::of(0);
        CHECK(RowStage::of(0) == stage && RowStage::of(3) != stage);
        const bool alone = std::thread::hardware_concurrency() < 2;  // no pool: the parts come one by one
        // A short upload while a part of a long one is held between its place and its copy.
        Rows longer((RowStage::kShortParts + 1) * RowStage::kPartRows, 1), shorter(RowStage::kPartRows + 3, 2);
        if (!alone) g_held = longer.got.data();
        std::thread first([&] { stage->upload(longer.f.data(), longer.n, longer.got.data(), nullptr); });
        {
            std::unique_lock<std::mutex> g(g_m);
            g_cv.wait(g, [&] { return g_holding || alone; });
        }
        // (Its parts take their places before the short one's.)
        while (!alone) {
            std::unique_lock<std::mutex> g(g_m);
            if (g_enqueued == RowStage::kShortParts) break;
            g.unlock();
            std::this_thread::yield();
        }
        std::atomic<bool> through{false};
        std::thread second([&] {
            stage->upload(shorter.f.data(), shorter.n, shorter.got.data(), nullptr);
            through = true;
        });
        for (int i = 0; i < 1000 && !through; i++) std::this_thread::sleep_for(std::chrono::milliseconds(10));
        CHECK(through);
        {
            std::lock_guard<std::mutex> g(g_m);
            g_held = nullptr;
            g_cv.notify_all();
        }
        first.join();
        second.join();
        drain();
        CHECK(longer.arrived() && shorter.arrived());

        // Twelve threads, uploads of all lengths.
        std::vector<std::thread> threads;
        std::atomic<int> wrong{0};
        for (unsigned t = 0; t < 12; t++)
            threads.emplace_back([&, t] {
                std::mt19937 rng(t);
                for (int k = 0; k < 20; k++) {
                    Rows r(1 + rng() % (k % 4 ? 200 : 1200), t * 100 + k);
                    stage->upload(r.f.data(), r.n, r.got.data(), nullptr);
                    drain();
                    wrong += !r.arrived();
                }
            });
        for (std::thread& t : threads) t.join();
        CHECK(wrong == 0);

        // A refused copy is reported, by long uploads and short ones, and later ones work.
        for (uint64_t n : {uint64_t(1), RowStage::kPartRows * 3, RowStage::kPartRows * 9}) {
            Rows r(n, 9);
            g_answer = cudaErrorInvalidValue;
            bool failed = false;
            try {
                stage->upload(r.f.data(), r.n, r.got.data(), nullptr);
            } catch (const bj::Fail&) {
                failed = true;
            }
            CHECK(failed);
            g_answer = cudaSuccess;
            stage->upload(r.f.data(), r.n, r.got.data(), nullptr);
            drain();
            CHECK(r.arrived());
        }
    }
    {
        std::lock_guard<std::mutex> g(g_m);
        g_stop = true;
        g_cv.notify_all();
    }
    engine.join();
    std::puts("ok");
    return 0;
}
