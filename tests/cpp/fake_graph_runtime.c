/* Stands in for the six graph calls of the CUDA runtime that sllm_graph_overlap makes: a chain of kernel nodes 1 .. n (node i's one predecessor is node i - 1; a node's
 * handle is its number, its kernel's too), every edge in one of three states, and the n-th call of a kind fails when asked to (tests/test_graph_overlap_cpu.py). */
#include <cuda_runtime_api.h>
#include <string.h>

enum { kMax = 16 };
static int nodes, edge_state[kMax + 1];                 /* 0 none, 1 ordinary, 2 programmatic */
static int calls_left[4];                               /* calls of a kind until one fails (0: never): look, remove, add, add and every later one */
void fake_reset(int n, int look, int remove, int add, int add_from) {
    nodes = n;
    for (int i = 2; i <= n; ++i) edge_state[i] = 1;
    calls_left[0] = look; calls_left[1] = remove; calls_left[2] = add; calls_left[3] = add_from;
}
int fake_edge(int node) { return edge_state[node]; }
static int fails(int kind) { return calls_left[kind] > 0 && --calls_left[kind] == 0; }

cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t* out, size_t* n) {
    (void)g;
    if (out)
        for (int i = 1; i <= nodes; ++i) out[i - 1] = (cudaGraphNode_t)(size_t)i;
    *n = (size_t)nodes;
    return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t node, enum cudaGraphNodeType* type) {
    (void)node;
    *type = cudaGraphNodeTypeKernel;
    return cudaSuccess;
}
cudaError_t cudaGraphKernelNodeGetParams(cudaGraphNode_t node, struct cudaKernelNodeParams* p) {
    memset(p, 0, sizeof *p);
    p->func = (void*)((size_t)node << 8);
    return cudaSuccess;
}
cudaError_t cudaGraphNodeGetDependencies_v2(cudaGraphNode_t node, cudaGraphNode_t* from, cudaGraphEdgeData* edge, size_t* n) {
    const size_t i = (size_t)node;
    if (fails(0)) return cudaErrorUnknown;
    if (from) {
        *from = (cudaGraphNode_t)(i - 1);
        memset(edge, 0, sizeof *edge);
        if (edge_state[i] == 2) {
            edge->type = cudaGraphDependencyTypeProgrammatic;
            edge->from_port = cudaGraphKernelNodePortProgrammatic;
        }
    }
    *n = i > 1 && edge_state[i] ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaGraphRemoveDependencies_v2(cudaGraph_t g, const cudaGraphNode_t* from, const cudaGraphNode_t* to, const cudaGraphEdgeData* edge, size_t n) {
    (void)g; (void)from; (void)edge; (void)n;
    if (fails(1)) return cudaErrorNotSupported;
    edge_state[(size_t)*to] = 0;
    return cudaSuccess;
}
cudaError_t cudaGraphAddDependencies_v2(cudaGraph_t g, const cudaGraphNode_t* from, const cudaGraphNode_t* to, const cudaGraphEdgeData* edge, size_t n) {
    (void)g; (void)from; (void)n;
    if (fails(2)) return cudaErrorNotSupported;
    if (calls_left[3] == 1) return cudaErrorNotSupported;
    if (calls_left[3] > 1) --calls_left[3];
    edge_state[(size_t)*to] = edge->type == cudaGraphDependencyTypeProgrammatic ? 2 : 1;
    return cudaSuccess;
}
