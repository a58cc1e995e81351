// Construction of CUDA graphs by capture.  A step that fails leaves no graph behind and the stream
// out of capture mode.
#pragma once

#include <cstddef>
#include <type_traits>

#include "errors.h"

namespace hw {

struct GraphHolder {
    cudaGraph_t g = nullptr;
    GraphHolder() = default;
    GraphHolder(const GraphHolder &) = delete;
    GraphHolder &operator=(const GraphHolder &) = delete;
    ~GraphHolder() {
        if (g) cudaGraphDestroy(g);
    }
};

// Captures what enqueue() puts on the stream into g, after its nodes deps[0..n).  enqueue returns a
// status, as this does.
template <class Enqueue>
int capture_into(cudaStream_t s, cudaGraph_t g, const cudaGraphNode_t *deps, size_t n, Enqueue enqueue) {
    HW_CUDA(cudaStreamBeginCaptureToGraph(s, g, deps, nullptr, n, cudaStreamCaptureModeThreadLocal));
    const int rc = enqueue();
    cudaGraph_t captured = nullptr;
    const cudaError_t e = cudaStreamEndCapture(s, &captured);
    if (rc != HW_OK || e != cudaSuccess) cudaGetLastError();  // a launch that failed during capture
    if (rc != HW_OK) return rc;
    HW_CUDA(e);
    return HW_OK;
}

// A WHILE or IF node with the handle `cond`, after deps[0..n); *body is its graph.
inline int add_conditional(cudaGraph_t g, const cudaGraphNode_t *deps, size_t n, cudaGraphConditionalHandle cond,
                           cudaGraphConditionalNodeType type, cudaGraphNode_t *node, cudaGraph_t *body) {
    cudaGraphNodeParams np = {cudaGraphNodeTypeConditional};
    np.conditional.handle = cond;
    np.conditional.type = type;
    np.conditional.size = 1;
    HW_CUDA(cudaGraphAddNode(node, g, deps, n, &np));
    *body = np.conditional.phGraph_out[0];
    return HW_OK;
}

// Loop graph of a CG: WHILE(status == running) { body } -> rest, where body(handle) enqueues one
// iteration whose last kernel sets the handle (loop_next), and rest() what follows the loop (if
// given); replaces *exec.
template <class Body, class Rest = std::nullptr_t>
int build_loop_graph(cudaStream_t s, cudaGraphExec_t *exec, Body body, Rest rest = nullptr) {
    if (*exec) cudaGraphExecDestroy(*exec);
    *exec = nullptr;
    int rc;
    GraphHolder G;
    HW_CUDA(cudaGraphCreate(&G.g, 0));
    cudaGraphConditionalHandle cond;
    HW_CUDA(cudaGraphConditionalHandleCreate(&cond, G.g, 1, cudaGraphCondAssignDefault));
    cudaGraphNode_t loop;
    cudaGraph_t inner;
    if ((rc = add_conditional(G.g, nullptr, 0, cond, cudaGraphCondTypeWhile, &loop, &inner)) != HW_OK) return rc;
    if ((rc = capture_into(s, inner, nullptr, 0, [&] { return body(cond), HW_OK; })) != HW_OK) return rc;
    if constexpr (!std::is_same<Rest, std::nullptr_t>::value)
        if ((rc = capture_into(s, G.g, &loop, 1, [&] { return rest(), HW_OK; })) != HW_OK) return rc;
    HW_CUDA(cudaGraphInstantiate(exec, G.g, 0));
    return HW_OK;
}

}  // namespace hw
