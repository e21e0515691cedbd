// csrc/runtime.cu — error reporting and device facts behind include/sllm_b200.h.
#include <atomic>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <unordered_map>
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
int g_tune_tc_polls = 1 << 24;   // tcgen05 kernels: 512 clocks apiece (4 seconds in all) after which a wait is given up
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

// Kernels launched through overlapping() and overlapping_alone(): sets that only grow, to at most as many as the library has instantiations; looked up on every launch, so
// without a lock.
struct KernelSet {
    static constexpr size_t kSlots = 1024;
    std::atomic<const void*> slots[kSlots];
    bool find(const void* kernel, bool add) {
        for (size_t i = reinterpret_cast<uintptr_t>(kernel) >> 4, n = 0; n < kSlots; ++i, ++n) {
            std::atomic<const void*>& slot = slots[i % kSlots];
            const void* held = slot.load(std::memory_order_acquire);
            if (held == nullptr && add && slot.compare_exchange_strong(held, kernel, std::memory_order_acq_rel)) return true;
            if (held == kernel) return true;      // compare_exchange has left what another thread put there
            if (held == nullptr && !add) return false;
        }
        return false;                             // a full table: this kernel's edges stay as they are
    }
};
static KernelSet g_overlap, g_overlap_alone;
void overlap_kernel(const void* kernel, bool alone) { (alone ? g_overlap_alone : g_overlap).find(kernel, true); }
static bool quiet(cudaError_t e) {               // a refusal that is no error of the caller's
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
}

// A captured graph as sllm_graph_overlap sees it.
struct StepGraph {
    struct Node {
        cudaGraphNode_t node;
        std::vector<size_t> from, to;        // predecessors, successors
        std::vector<cudaGraphEdgeData> edges;    // from its predecessors
        bool kernel = false, waits = false;  // waits: a kernel that may become resident early
        size_t before = 0, after = 0;        // nodes that have to complete before it, nodes that wait for it
    };
    std::vector<Node> nodes;
    bool read(cudaGraph_t g);
    int overlap(cudaGraph_t g, size_t i) const;
    int separate(cudaGraph_t g, size_t i) const;
};

bool StepGraph::read(cudaGraph_t g) {        // false: the runtime will not say all of it
    size_t n = 0;
    if (!quiet(cudaGraphGetNodes(g, nullptr, &n))) return false;
    std::vector<cudaGraphNode_t> handles(n);
    if (!quiet(cudaGraphGetNodes(g, handles.data(), &n))) return false;
    std::unordered_map<cudaGraphNode_t, size_t> index;
    for (size_t i = 0; i < n; ++i) index[handles[i]] = i;
    nodes.resize(n);
    for (size_t i = 0; i < n; ++i) {
        Node& x = nodes[i];
        x.node = handles[i];
        size_t deps = 0;
        if (!quiet(cudaGraphNodeGetDependencies_v2(x.node, nullptr, nullptr, &deps))) return false;
        std::vector<cudaGraphNode_t> from(deps);
        x.edges.resize(deps);
        if (deps && !quiet(cudaGraphNodeGetDependencies_v2(x.node, from.data(), x.edges.data(), &deps))) return false;
        for (size_t k = 0; k < deps; ++k) {
            const auto at = index.find(from[k]);
            if (at == index.end()) return false;
            x.from.push_back(at->second);
            nodes[at->second].to.push_back(i);
        }
        cudaGraphNodeType type;
        if (!quiet(cudaGraphNodeGetType(x.node, &type))) return false;
        x.kernel = type == cudaGraphNodeTypeKernel;
        cudaKernelNodeParams p{};
        if (!x.kernel || !quiet(cudaGraphKernelNodeGetParams(x.node, &p))) continue;     // or another library's kernel
        x.waits = g_overlap.find(p.func, false) || (g_overlap_alone.find(p.func, false) && (size_t)p.gridDim.x * p.gridDim.y * p.gridDim.z == 1);
    }
    // how many nodes each one follows: a row of bits per node, predecessors first; every node it follows is followed by it
    const size_t words = (n + 63) / 64;
    std::vector<uint64_t> bits(n * words, 0);
    std::vector<size_t> order, open(n);
    for (size_t i = 0; i < n; ++i)
        if ((open[i] = nodes[i].from.size()) == 0) order.push_back(i);
    for (size_t k = 0; k < order.size(); ++k) {
        const size_t i = order[k];
        for (size_t w = 0; w < words; ++w)
            for (uint64_t rest = bits[i * words + w]; rest; rest &= rest - 1) {
                ++nodes[i].before;
                ++nodes[w * 64 + __builtin_ctzll(rest)].after;
            }
        for (size_t j : nodes[i].to) {
            for (size_t w = 0; w < words; ++w) bits[j * words + w] |= bits[i * words + w];
            bits[j * words + i / 64] |= uint64_t(1) << (i % 64);
            if (--open[j] == 0) order.push_back(j);
        }
    }
    return true;
}

// One edge for another: 1 = done; 0 = as it was, since the runtime will not exchange it; -1 = lost.
static int exchange(cudaGraph_t g, cudaGraphNode_t from, cudaGraphNode_t to, const cudaGraphEdgeData& old, const cudaGraphEdgeData& edge) {
    if (!quiet(cudaGraphRemoveDependencies_v2(g, &from, &to, &old, 1))) return 0;
    if (quiet(cudaGraphAddDependencies_v2(g, &from, &to, &edge, 1))) return 1;
    return quiet(cudaGraphAddDependencies_v2(g, &from, &to, &old, 1)) ? 0 : -1;
}

// The edge in front of node i made programmatic: as exchange(), 0 also where it has to stay.
int StepGraph::overlap(cudaGraph_t g, size_t i) const {
    const Node& x = nodes[i];
    // One predecessor, a kernel with no other successor, and no node in a parallel branch of the step (every other one completes before it or waits for it): its own wait takes the
    // place of the edge, as between two launches of one stream. Where there are branches a CTA that only waits keeps another branch's off its SM. Measured, us a step of Nelutar,
    // whose layers have branches, edges as captured | exchanged there too | only outside: width 1024, one request 388 | 368 | 376, four 503 | 503 | 491, eight 689 | 713 | 677;
    // width 2048 537 | 498 | 525, 893 | 975 | 880, 1443 | 1490 | 1430; and at nine requests replays with edges exchanged there came to a stand.
    if (!x.waits || x.from.size() != 1 || x.edges[0].type != cudaGraphDependencyTypeDefault || x.edges[0].from_port != cudaGraphKernelNodePortDefault) return 0;
    const Node& previous = nodes[x.from[0]];
    if (!previous.kernel || previous.to.size() != 1 || x.before + x.after + 1 != nodes.size()) return 0;
    cudaGraphEdgeData early{};
    early.type = cudaGraphDependencyTypeProgrammatic;
    early.from_port = cudaGraphKernelNodePortProgrammatic;
    return exchange(g, previous.node, x.node, x.edges[0], early);
}

// Programmatic edges that the capture itself has made (products are launched with that attribute) from one branch to another, made ordinary: a launch at the start of a branch or behind
// a join is not one behind another in a stream either. 0 or -1.
int StepGraph::separate(cudaGraph_t g, size_t i) const {
    const Node& x = nodes[i];
    for (size_t k = 0; k < x.from.size(); ++k) {
        if (x.edges[k].type != cudaGraphDependencyTypeProgrammatic || (x.from.size() == 1 && nodes[x.from[k]].to.size() == 1)) continue;
        if (exchange(g, nodes[x.from[k]].node, x.node, x.edges[k], cudaGraphEdgeData{}) < 0) return -1;
    }
    return 0;
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
    StepGraph step;
    if (step.read(g)) {
        for (size_t i = 0; i < step.nodes.size(); ++i) {
            const int done = step.separate(g, i) < 0 ? -1 : step.overlap(g, i);
            SLLM_REQUIRE(done >= 0, SLLM_ESTATE, "graph_overlap: the runtime took an edge and would not have it back; the graph has to be captured again");
            changed += done;
        }
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
