// launch_after (csrc/after.cuh) on a CUDA runtime of the test's own: the launch it makes, and the status it hands back.
#include <cuda_runtime.h>

#include <cstdio>

inline void cudaGridDependencySynchronize() {}
inline void cudaTriggerProgrammaticLaunchCompletion() {}

static cudaError_t g_answer = cudaSuccess;
static cudaLaunchConfig_t g_config;
static int g_first = 0;
static long g_second = 0;

template <typename... P>
cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* c, void (*)(P...), int a, long b) {
    g_config = *c;
    g_first = a;
    g_second = b;
    return g_answer;
}

#include "after.cuh"

static void kernel(int, long) {}

#define CHECK(x)                                                  \
    if (!(x)) {                                                   \
        std::printf("line %d: %s does not hold\n", __LINE__, #x); \
        return 1;                                                 \
    }

int main() {
    CHECK(bj::launch_after(kernel, dim3(7, 2), 128, 60'000, nullptr, 3, 4) == cudaSuccess);
    CHECK(g_config.gridDim.x == 7 && g_config.gridDim.y == 2 && g_config.blockDim.x == 128);
    CHECK(g_config.dynamicSmemBytes == 60'000 && g_config.numAttrs == 1 && g_first == 3 && g_second == 4);
    for (cudaError_t e : {cudaErrorInvalidValue, cudaErrorLaunchOutOfResources, cudaErrorInvalidDeviceFunction}) {
        g_answer = e;
        CHECK(bj::launch_after(kernel, 1, 1, 0, nullptr, 1, 1) == e);
    }
    std::puts("ok");
    return 0;
}
