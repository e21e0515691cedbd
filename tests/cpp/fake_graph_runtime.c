/* Stands in for the calls about graphs that sllm_graph_overlap makes: kernel nodes 1 .. n whose handle is their number (their kernel's address 256 times it), a
 * chain unless fake_from says otherwise. Every edge is in one of three states, the n-th call of a kind fails when asked to, and a kernel may have several CTAs
 * (tests/test_graph_overlap_cpu.py). */
#include <cuda_runtime_api.h>
#include <string.h>

enum { kMax = 16 };
static int nodes, from[kMax + 1][2], edge_state[kMax + 1][2];   /* up to two predecessors; 0 no edge, 1 ordinary, 2 programmatic */
static int ctas[kMax + 1];
static int calls_left[4];                                       /* calls of a kind until one fails (0: never): look, remove, add, add and every later one */
void fake_reset(int n, int look, int remove, int add, int add_from) {
    nodes = n;
    memset(from, 0, sizeof from);
    memset(edge_state, 0, sizeof edge_state);
    for (int i = 1; i <= n; ++i) {
        from[i][0] = i - 1;
        edge_state[i][0] = i > 1;
        ctas[i] = 1;
    }
    calls_left[0] = look; calls_left[1] = remove; calls_left[2] = add; calls_left[3] = add_from;
}
void fake_from(int node, int a, int a_state, int b, int b_state) {
    from[node][0] = a; edge_state[node][0] = a_state;
    from[node][1] = b; edge_state[node][1] = b_state;
}
void fake_grid(int node, int grid) { ctas[node] = grid; }
int fake_edge(int node, int k) { return edge_state[node][k]; }
static int fails(int kind) { return calls_left[kind] > 0 && --calls_left[kind] == 0; }
static int* state_of(const cudaGraphNode_t* a, const cudaGraphNode_t* to) {
    const size_t i = (size_t)*to;
    return &edge_state[i][from[i][0] == (int)(size_t)*a ? 0 : 1];
}

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
    const size_t i = (size_t)node;
    memset(p, 0, sizeof *p);
    p->func = (void*)(i << 8);
    p->gridDim.x = (unsigned)ctas[i]; p->gridDim.y = p->gridDim.z = 1;
    return cudaSuccess;
}
cudaError_t cudaGraphNodeGetDependencies_v2(cudaGraphNode_t node, cudaGraphNode_t* out, cudaGraphEdgeData* edge, size_t* n) {
    const size_t i = (size_t)node;
    size_t k = 0;
    if (fails(0)) return cudaErrorUnknown;
    for (int j = 0; j < 2; ++j) {
        if (edge_state[i][j] == 0) continue;
        if (out) {
            out[k] = (cudaGraphNode_t)(size_t)from[i][j];
            memset(edge + k, 0, sizeof *edge);
            if (edge_state[i][j] == 2) {
                edge[k].type = cudaGraphDependencyTypeProgrammatic;
                edge[k].from_port = cudaGraphKernelNodePortProgrammatic;
            }
        }
        ++k;
    }
    *n = k;
    return cudaSuccess;
}
cudaError_t cudaGraphRemoveDependencies_v2(cudaGraph_t g, const cudaGraphNode_t* a, const cudaGraphNode_t* to, const cudaGraphEdgeData* edge, size_t n) {
    (void)g; (void)edge; (void)n;
    if (fails(1)) return cudaErrorNotSupported;
    *state_of(a, to) = 0;
    return cudaSuccess;
}
cudaError_t cudaGraphAddDependencies_v2(cudaGraph_t g, const cudaGraphNode_t* a, const cudaGraphNode_t* to, const cudaGraphEdgeData* edge, size_t n) {
    (void)g; (void)n;
    if (fails(2)) return cudaErrorNotSupported;
    if (calls_left[3] == 1) return cudaErrorNotSupported;
    if (calls_left[3] > 1) --calls_left[3];
    *state_of(a, to) = edge->type == cudaGraphDependencyTypeProgrammatic ? 2 : 1;
    return cudaSuccess;
}
