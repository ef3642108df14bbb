// bj::capture_graph (csrc/graphs.cpp) on a CUDA runtime and an executor of the test's own: whatever the executor throws
// while it is captured, the capture ends, the context takes calls again and the query is left to plain execution.
#include "engine.h"

#include <cstdio>
#include <cstdlib>
#include <new>
#include <stdexcept>

static int g_throw = 0;
static bool g_capturing = false;
static int g_synced = 0;

namespace bj {
bool capture_graph(bj_context*, GraphEntry&, const bj_plan*, bj_resident* const*, int);

void phase_stats(const std::vector<cudaEvent_t>&, bj_stats&) {}
bool run_pipelines(bj_context* ctx, const ExecPlan&, const std::vector<const DevTable*>&, bj_result&, int, uint64_t&) {
    ctx->prof_events.push_back(nullptr);
    switch (g_throw) {
        case 0: throw Fail{BJ_ERR_OOM, "device"};
        case 1: throw std::runtime_error("a launch was refused");
        case 2: throw std::length_error("result pages beyond one launch");
        default: throw std::bad_alloc();
    }
}
int execute_common(bj_context*, const bj_plan*, bj_resident* const*, int, bj_result**, bool) { return BJ_ERR_INTERNAL; }
int fail_to_status(bj_context*, const Fail& f) { return f.status; }
int make_exec_plan(const bj_plan&, ExecPlan& out, std::string&, bool, const std::vector<double>*, PlanSpace) {
    out.empty = false;
    return BJ_OK;
}
void collect_columns(const ExecPlan&, uint32_t, uint64_t, std::vector<uint8_t>&) {}
PlanSpace plan_space_default() { return PlanSpace::Auto; }
TuneConfig tune_for(const bj_context*, const ExecPlan&) { return TuneConfig{}; }
} // namespace bj

extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    g_capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    g_capturing = false;
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    g_synced++;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void**, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
}

#define CHECK(x)                                                                    \
    if (!(x)) {                                                                     \
        std::printf("throw %d, line %d: %s does not hold\n", g_throw, __LINE__, #x); \
        return 1;                                                                   \
    }

int main() {
    bj_plan plan{};
    for (g_throw = 0; g_throw < 4; g_throw++) {
        bj_context ctx;
        bj::GraphEntry g;
        g_synced = 0;
        bool captured = true;
        try {
            captured = bj::capture_graph(&ctx, g, &plan, nullptr, 0);
        } catch (...) {
            std::printf("throw %d leaves capture_graph, the stream %s\n", g_throw, g_capturing ? "still captured" : "free");
            return 1;
        }
        CHECK(!captured && !g.exec);
        CHECK(!g_capturing && g_synced > 0);
        CHECK(ctx.tape_mode == 0 && !ctx.tape && !ctx.graph_output && ctx.prof_events.empty());
    }
    std::puts("ok");
    return 0;
}
