// Graph construction (hila_b200/csrc/graph_build.h) over a fake CUDA runtime: whichever call fails,
// the status says so, every graph that was made is destroyed, the stream is not left capturing, and
// no executable graph stays behind.  No GPU involved.
#include <cstdarg>
#include <cstdio>

#include "graph_build.h"

namespace {
int calls, fail_at, graphs, execs, capturing;
cudaError_t step() { return ++calls == fail_at ? cudaErrorUnknown : cudaSuccess; }
int made;
}  // namespace

extern "C" {
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) graphs++, *g = (cudaGraph_t)&made;
    return e;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return graphs--, cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) {
    *h = 1;
    return step();
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t, cudaGraphNodeParams *p) {
    static cudaGraph_t inner;
    p->conditional.phGraph_out = &inner;
    return step();
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *,
                                          size_t, cudaStreamCaptureMode) {
    const cudaError_t e = step();
    if (e == cudaSuccess) capturing++;
    return e;
}
// an invalid capture ends with an error and without a graph, but it ends
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return capturing--, *g = nullptr, step(); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
    const cudaError_t e = step();
    if (e == cudaSuccess) execs++, *x = (cudaGraphExec_t)&made;
    return e;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return execs--, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
}
void hw::set_error(const char *, ...) {}

int main() {
    int failures = 0, total = 0;
    for (fail_at = 0; fail_at == 0 || fail_at <= total; fail_at++) {
        calls = graphs = execs = capturing = 0;
        int bodies = 0, rests = 0;
        cudaGraphExec_t exec = nullptr;
        const int rc = hw::build_loop_graph(
            nullptr, &exec, [&](cudaGraphConditionalHandle) { bodies++; }, [&] { rests++; });
        if (fail_at == 0) total = calls;
        const bool ok = fail_at == 0 ? rc == HW_OK && exec && execs == 1 && bodies == 1 && rests == 1
                                     : rc == HW_ERR_CUDA && !exec && execs == 0;
        if (!ok || graphs != 0 || capturing != 0) {
            std::printf("FAILED with call %d: status %d, %d graphs, capturing %d\n", fail_at, rc, graphs, capturing);
            failures++;
        }
    }
    // what is enqueued may fail, too
    capturing = fail_at = 0;
    if (hw::capture_into(nullptr, nullptr, nullptr, 0, [] { return (int)HW_ERR_OOM; }) != HW_ERR_OOM || capturing)
        failures++;
    if (total < 8) failures++;
    if (failures == 0) std::printf("graph construction passed\n");
    return failures;
}
