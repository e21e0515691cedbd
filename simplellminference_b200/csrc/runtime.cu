// csrc/runtime.cu — error reporting and device facts behind include/sllm_b200.h.
#include <atomic>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace sllm {

static thread_local char g_err[512] = "";
thread_local int64_t g_launches = 0;
int g_tune_ctas_per_sm = 0;
int g_tune_pf_bn = 0;   // prefill GEMM: force the N tile (128 / 256), 0 = heuristic
int g_tune_pf_pdl = 1;     // prefill kernels: programmatic dependent launch (set-up overlaps the previous kernel's tail)
int g_tune_pf_ksplit = -1;  // prefill GEMM, residual epilogue: 0 = never split K, n > 0 = up to n parts, -1 = heuristic (up to 4)
int g_tune_batch_graph = 0;   // batched decode: 1 = replay one CUDA graph per live-slot count instead of the launch sequence (experimental)
int g_tune_batch_rows4 = 0;   // batched decode GEMV: 1 = four weight rows per warp at a time for >= 3 vectors (experimental)
int g_tune_batch_ksplit = 0;  // batched decode, with rows4: down projection with K cut in two over grid.y when more vectors are live than fit whole rows (experimental)
int g_tune_mega_debug = 0;   // decode megakernel measurement aid (MegaParams::debug): bit 0 = no grid barriers, bit 1 = no dot products; results are garbage
int g_tune_seq_attn_mma = 1;   // ragged-batch attention: 1 = tensor-core body for bf16 pools on steps with prompt portions, 0 = always the fp32 body
int g_tune_tc_polls = 1 << 24;   // tcgen05 attention kernels: polls after which a wait is given up
int g_tune_pf_pair = -1;   // prefill GEMM: 1 / 0 = force / forbid the two-SM (cta_group::2) kernel, -1 = heuristic

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    set_error("CUDA error %d (%s) at %s:%d in %s", (int)e, cudaGetErrorString(e), file, line, what);
    return (int)e;
}

int32_t* g_status = nullptr;

int status_word(int32_t** word) {
    static std::mutex lock;
    std::lock_guard<std::mutex> hold(lock);
    if (!g_status) {
        // an allocation would end a capture that runs in this thread; this one takes no part in it
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        SLLM_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        void* p = nullptr;
        const cudaError_t e = cudaHostAlloc(&p, sizeof(int32_t), cudaHostAllocMapped | cudaHostAllocPortable);
        cudaThreadExchangeStreamCaptureMode(&mode);
        SLLM_CUDA(e);
        *static_cast<int32_t*>(p) = 0;
        g_status = static_cast<int32_t*>(p);      // unified addressing: the same address on every device
    }
    *word = g_status;
    return SLLM_OK;
}

int status_take() {
    const int32_t what = g_status ? __atomic_exchange_n(g_status, 0, __ATOMIC_ACQ_REL) : 0;
    if (what == 0) return SLLM_OK;
    SLLM_REQUIRE(what != kStatusBatch, SLLM_EINVAL, "seq_ssd_blocks: n_qtiles of an earlier launch does not count the tiles of all its tokens; its results are incomplete");
    set_error("a kernel gave up waiting for its copies or products: the results of an earlier launch are incomplete");
    return SLLM_ETIMEOUT;
}

// Kernels launched through overlapping(): a set that only grows, to at most as many as the library has instantiations; looked up on every launch, so without a lock.
static constexpr size_t kOverlapSlots = 1024;
static std::atomic<const void*> g_overlap[kOverlapSlots];
static bool overlap_find(const void* kernel, bool add) {
    for (size_t i = reinterpret_cast<uintptr_t>(kernel) >> 4, n = 0; n < kOverlapSlots; ++i, ++n) {
        std::atomic<const void*>& slot = g_overlap[i % kOverlapSlots];
        const void* held = slot.load(std::memory_order_acquire);
        if (held == nullptr && add && slot.compare_exchange_strong(held, kernel, std::memory_order_acq_rel)) return true;
        if (held == kernel) return true;      // compare_exchange has left what another thread put there
        if (held == nullptr && !add) return false;
    }
    return false;                             // a full table: this kernel's edges stay as they are
}
void overlap_kernel(const void* kernel) { overlap_find(kernel, true); }
static bool quiet(cudaError_t e) {               // a refusal that is no error of the caller's
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
}
// The edge in front of one node: 1 = programmatic now; 0 = as it was, being of another kind or because the runtime will not exchange it; -1 = lost.
static int overlap_edge(cudaGraph_t g, cudaGraphNode_t node) {
    cudaGraphNodeType type;
    if (!quiet(cudaGraphNodeGetType(node, &type)) || type != cudaGraphNodeTypeKernel) return 0;
    cudaKernelNodeParams p{};
    if (!quiet(cudaGraphKernelNodeGetParams(node, &p)) || !overlap_find(p.func, false)) return 0;     // another library's kernel, or one that does not wait
    // One predecessor, a kernel: this node's own wait takes the place of the edge. Joins of several branches keep theirs (a step of Nelutar measured the same with
    // those converted too).
    size_t deps = 0;
    if (!quiet(cudaGraphNodeGetDependencies_v2(node, nullptr, nullptr, &deps)) || deps != 1) return 0;
    cudaGraphNode_t from = nullptr;
    cudaGraphEdgeData edge{}, early{};
    if (!quiet(cudaGraphNodeGetDependencies_v2(node, &from, &edge, &deps)) || !quiet(cudaGraphNodeGetType(from, &type))) return 0;
    if (type != cudaGraphNodeTypeKernel || edge.type != cudaGraphDependencyTypeDefault || edge.from_port != cudaGraphKernelNodePortDefault) return 0;
    early.type = cudaGraphDependencyTypeProgrammatic;
    early.from_port = cudaGraphKernelNodePortProgrammatic;
    if (!quiet(cudaGraphRemoveDependencies_v2(g, &from, &node, &edge, 1))) return 0;
    if (quiet(cudaGraphAddDependencies_v2(g, &from, &node, &early, 1))) return 1;
    return quiet(cudaGraphAddDependencies_v2(g, &from, &node, &edge, 1)) ? 0 : -1;
}

int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

int smem_optin_bytes() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (n <= 0) n = 48 * 1024;
    }
    return n;
}

}  // namespace sllm

extern "C" {

const char* sllm_last_error(void) { return sllm::g_err; }
int sllm_status(void) { return sllm::status_check(); }
int sllm_abi_version(void) { return 1; }

int sllm_tune(int32_t key, int32_t value) {
    switch (key) {
        case 0: sllm::g_tune_ctas_per_sm = value; return SLLM_OK;
        case 1: sllm::g_tune_pf_bn = value; return SLLM_OK;
        case 2: sllm::g_tune_pf_pair = value; return SLLM_OK;
        case 3: sllm::g_tune_pf_pdl = value; return SLLM_OK;
        case 4: sllm::g_tune_pf_ksplit = value; return SLLM_OK;
        case 5: sllm::g_tune_batch_graph = value; return SLLM_OK;
        case 6: sllm::g_tune_batch_rows4 = value; return SLLM_OK;
        case 7: sllm::g_tune_batch_ksplit = value; return SLLM_OK;
        case 8: sllm::g_tune_mega_debug = value; return SLLM_OK;
        case 9: sllm::g_tune_seq_attn_mma = value; return SLLM_OK;
        case 10:
            SLLM_REQUIRE(value >= 0, SLLM_EINVAL, "a limit of %d polls", value);
            sllm::g_tune_tc_polls = value;
            return SLLM_OK;
        default: sllm::set_error("unknown tunable %d", key); return SLLM_EINVAL;
    }
}

int sllm_graph_overlap(void* graph, int32_t* edges) {
    using namespace sllm;
    SLLM_REQUIRE(graph, SLLM_EINVAL, "graph_overlap: no graph");
    const cudaGraph_t g = reinterpret_cast<cudaGraph_t>(graph);
    int32_t changed = 0;
    size_t n = 0;
    SLLM_CUDA(cudaGraphGetNodes(g, nullptr, &n));
    std::vector<cudaGraphNode_t> nodes(n);
    SLLM_CUDA(cudaGraphGetNodes(g, nodes.data(), &n));
    for (size_t i = 0; i < n; ++i) {
        const int done = overlap_edge(g, nodes[i]);
        SLLM_REQUIRE(done >= 0, SLLM_ESTATE, "graph_overlap: the runtime took an edge and would not have it back; the graph has to be captured again");
        changed += done;
    }
    if (edges) *edges = changed;
    return SLLM_OK;
}

int sllm_device_info(int32_t* sms, int32_t* smem, size_t* total, size_t* free_) {
    int n = 0;
    SLLM_CUDA(cudaGetDeviceCount(&n));
    SLLM_REQUIRE(n > 0, SLLM_ESTATE, "no CUDA device visible: libsllm_b200 has no CPU fallback");
    if (sms) *sms = sllm::sm_count();
    if (smem) *smem = sllm::smem_optin_bytes();
    size_t f = 0, t = 0;
    SLLM_CUDA(cudaMemGetInfo(&f, &t));
    if (total) *total = t;
    if (free_) *free_ = f;
    return SLLM_OK;
}

}  // extern "C"
