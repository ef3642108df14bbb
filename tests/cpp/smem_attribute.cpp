// The bookkeeping of allow_smem (csrc/smem.h) on a CUDA runtime of the test's own: which calls set the attribute, with
// what, when they succeed and when they fail.
#include "smem.h"

#include <cstdio>
#include <map>
#include <utility>

static thread_local int g_device = 0;
static cudaError_t g_answer = cudaSuccess;
static std::atomic<int> g_calls{0};
static std::map<std::pair<const void*, int>, int> g_set;  // (kernel, device) -> bytes

extern "C" cudaError_t cudaGetDevice(int* d) {
    *d = g_device;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    g_calls++;
    if (g_answer == cudaSuccess && a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_set[{f, g_device}] = v;
    return g_answer;
}

static void one(int) {}
static void two(float) {}

#define CHECK(x)                                              \
    if (!(x)) {                                               \
        std::printf("line %d: %s does not hold\n", __LINE__, #x); \
        return 1;                                             \
    }

int main() {
    const void* f1 = reinterpret_cast<const void*>(&one);
    const void* f2 = reinterpret_cast<const void*>(&two);
    // Every device and kernel gets its own, once.
    for (int round = 0; round < 3; round++)
        for (int d : {0, 1, 7, 63}) {
            g_device = d;
            CHECK(bj::allow_smem<one>(80'000) == cudaSuccess);
            CHECK(bj::allow_smem<two>(70'000) == cudaSuccess);
        }
    CHECK(g_calls == 8);
    for (int d : {0, 1, 7, 63}) CHECK((g_set[{f1, d}] == 80'000 && g_set[{f2, d}] == 70'000));
    // A refusal is reported, and tried again by the next launch.
    g_device = 2;
    g_answer = cudaErrorInvalidValue;
    CHECK(bj::allow_smem<one>(80'000) == cudaErrorInvalidValue);
    CHECK(bj::allow_smem<one>(80'000) == cudaErrorInvalidValue);
    g_answer = cudaSuccess;
    CHECK(bj::allow_smem<one>(80'000) == cudaSuccess && g_calls == 11);
    CHECK(bj::allow_smem<one>(80'000) == cudaSuccess && g_calls == 11);
    // Devices beyond the bits are set each time.
    for (int d : {64, 65}) {
        g_device = d;
        CHECK(bj::allow_smem<one>(80'000) == cudaSuccess);
        CHECK((g_set[{f1, d}] == 80'000));
    }
    CHECK(g_calls == 13);
    std::puts("ok");
    return 0;
}
