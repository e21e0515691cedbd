// csrc/gemv.cu — sllm_gemv: the plain (unfused) decode GEMV behind kernel::matmul_kernel_cuda.
#include "gemv_core.cuh"

namespace sllm {

struct PlainPolicy {
    const float* x;
    const void* W_;
    const float* sc;
    float* y;
    int grp, nrows, ncols;
    float scale;
    __device__ int units() const { return (nrows + 1) >> 1; }
    __device__ void rows(int u, int64_t& r0, int64_t& r1) const { r0 = 2 * (int64_t)u; r1 = min(2 * u + 1, nrows - 1); }
    __device__ const void* W() const { return W_; }
    __device__ const float* scales() const { return sc; }
    __device__ int group() const { return grp; }
    __device__ int cols() const { return ncols; }
    template <int WD> __device__ void stage_t(float* xs, float*) const { stage_x_plain<WD>(xs, x, ncols); }
    __device__ void emit(int u, float s0, float s1) const {
        y[2 * u] = s0 * scale;  // (sum) * scale, matmul_kernel.cpp:26
        if (2 * u + 1 < nrows) y[2 * u + 1] = s1 * scale;
    }
};

template <int WD>
struct PlainPolicyT : PlainPolicy {
    __device__ void stage(float* xs, float* red) const { this->template stage_t<WD>(xs, red); }
};

template <int WD>
__global__ void __launch_bounds__(kGemvThreads) gemv_plain_kernel(PlainPolicyT<WD> pol) { gemv_body<WD>(pol); }

// Few rows: `parts` (2, 4 or 8) neighbouring warps cut the columns of a pair of rows among themselves, so that all of the matrix is asked for at once where a warp per pair leaves SMs
// without work and takes its rows in several trips. Bound: the latency of one trip behind the launch. The partial sums meet in shared memory in a fixed order.
template <int WD>
__global__ void __launch_bounds__(kGemvThreads, 2) gemv_split_kernel(PlainPolicyT<WD> pol, int parts, int group_shift) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float2 part_sum[kGemvWarps];
    constexpr int E = WInfo<WD>::E;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % parts;
    const int unit = (blockIdx.x * kGemvWarps + warp) / parts;
    const int nchunks = pol.ncols / E, per = (nchunks + parts - 1) / parts, lo = part * per, hi = min(nchunks, lo + per);
    const int cpg = WD == SLLM_INT8 ? pol.grp / 16 : 1, groups = WD == SLLM_INT8 ? pol.ncols / pol.grp : 0;
    const bool live = unit < pol.units();
    int64_t r0 = 0, r1 = 0;
    if (live) pol.rows(unit, r0, r1);
    const uint4 *w0 = reinterpret_cast<const uint4*>(pol.W_) + r0 * nchunks, *w1 = reinterpret_cast<const uint4*>(pol.W_) + r1 * nchunks;
    const float *sc0 = pol.sc + r0 * groups, *sc1 = pol.sc + r1 * groups;
    Batch<WD> cur;
    auto load = [&](int base) {
#pragma unroll
        for (int u = 0; u < kGemvU; ++u) {
            const int c = base + u * 32 + lane;
            const bool has = live && c < hi;
            cur.w0[u] = has ? ldg_stream(w0 + c) : make_uint4(0, 0, 0, 0);
            cur.w1[u] = has ? ldg_stream(w1 + c) : make_uint4(0, 0, 0, 0);
            if (WD == SLLM_INT8) {
                const int g = group_shift >= 0 ? c >> group_shift : c / cpg;
                cur.s0[u] = has ? __ldg(sc0 + g) : 0.0f;
                cur.s1[u] = has ? __ldg(sc1 + g) : 0.0f;
            }
        }
    };
    load(lo);
    pol.stage(smem, smem + pol.ncols);
    __syncthreads();
    const float4* xs4 = reinterpret_cast<const float4*>(smem);
    float a0 = 0.0f, a1 = 0.0f;
    for (int base = lo; base < hi; base += 32 * kGemvU) {
#pragma unroll
        for (int u = 0; u < kGemvU; ++u) {
            const int c = base + u * 32 + lane;
            if (c < hi) {
                if (WD == SLLM_INT8) {
                    a0 = fmaf(chunk_dot<WD>(cur.w0[u], xs4, c, nchunks, 0.0f), cur.s0[u], a0);
                    a1 = fmaf(chunk_dot<WD>(cur.w1[u], xs4, c, nchunks, 0.0f), cur.s1[u], a1);
                } else {
                    a0 = chunk_dot<WD>(cur.w0[u], xs4, c, nchunks, a0);
                    a1 = chunk_dot<WD>(cur.w1[u], xs4, c, nchunks, a1);
                }
            }
        }
        if (base + 32 * kGemvU < hi) load(base + 32 * kGemvU);
    }
    a0 = warp_sum(a0);
    a1 = warp_sum(a1);
    if (lane == 0) part_sum[warp] = make_float2(a0, a1);
    __syncthreads();
    if (live && part == 0 && lane == 0) {
        for (int i = 1; i < parts; ++i) {
            a0 += part_sum[warp + i].x;
            a1 += part_sum[warp + i].y;
        }
        pol.emit(unit, a0, a1);
    }
}

constexpr size_t kCtaSharedReserve = 1024;      // what the system keeps of an SM's shared memory for every resident CTA

template <int WD>
static int launch_plain(const PlainPolicy& p, cudaStream_t st) {
    const size_t smem = gemv_smem_bytes(p.ncols);
    static size_t configured = 0;
    if (smem > 48 * 1024 && smem > configured) {
        SLLM_REQUIRE(smem <= (size_t)smem_optin_bytes(), SLLM_ENOTSUP, "gemv: cols=%d does not fit shared memory", p.ncols);
        SLLM_CUDA(cudaFuncSetAttribute(gemv_plain_kernel<WD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    PlainPolicyT<WD> pt;
    static_cast<PlainPolicy&>(pt) = p;
    // More warps a pair of rows while all CTAs are resident at once and a warp keeps enough columns: the sums' way through shared memory costs 0.3 us, and a second CTA an SM, which stages the vector again,
    // another 0.2 (int8 0.5). Measured in a captured graph, us, a warp per pair | 2, 4 and 8: fp32 256 x 512 2.3 | 2.5 2.5 2.6, 256 x 1024 2.6 | 2.6 2.5 2.6, 700 x 1024 2.7 | 2.6 2.9, 2048 x 1024 3.7 | 3.6, 500 x 4096 7.2 | 4.9 3.7 3.7,
    // 2048 x 5632 12.2 | 10.2; bf16 500 x 1024 2.5 | 2.5 2.6 2.9, 2048 x 1024 3.0 | 3.1, 2048 x 1536 3.7 | 3.5, 700 x 2048 3.2 | 2.9 3.1, 256 x 4096 4.2 | 3.0 2.8 2.8, 2048 x 5632 8.5 | 7.1; int8 256 x 1024 2.8 | 2.9 3.0 3.0, 256 x 2048 3.5 | 3.2
    // 3.1 3.2, 700 x 2048 3.5 | 3.2 3.7, 1200 x 2048 3.5 | 3.9, 2048 x 4096 4.9 | 5.2, 500 x 5632 6.2 | 4.4 3.9 4.6, 2048 x 5632 6.9 | 6.5 (a call of it 8.20 | 8.16: the launch and the host). One warp a pair from 2369 rows on.
    // A vector that takes more than half of an SM's shared memory (28 700 columns) leaves it one CTA, and one that fills it no room for the partial sums beside it.
    const size_t split_smem = smem + kGemvWarps * sizeof(float2), sm_smem = (size_t)smem_optin_bytes() + kCtaSharedReserve;
    const int resident = 2 * (split_smem + kCtaSharedReserve) <= sm_smem ? 2 : split_smem + kCtaSharedReserve <= sm_smem ? 1 : 0;
    const int units = (p.nrows + 1) / 2, chunks = p.ncols / WInfo<WD>::E, warps = resident * kGemvWarps * sm_count();
    constexpr bool kInt8 = WD == SLLM_INT8;
    int parts = 1;
    while (parts < kGemvWarps && 2LL * parts * units <= warps && chunks >= (kInt8 ? 128 : 192)) {
        const bool second = 2LL * parts * units > kGemvWarps * sm_count();
        if (chunks / (2 * parts) < (second ? (kInt8 ? 160 : 96) : (kInt8 ? 32 : 64))) break;
        parts *= 2;
    }
    if (parts > 1 && g_tune_ctas_per_sm == 0) {
        static size_t split_configured = 0;
        if (split_smem > 48 * 1024 && smem > split_configured) {
            SLLM_CUDA(cudaFuncSetAttribute(gemv_split_kernel<WD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            split_configured = smem;
        }
        const int cpg = WD == SLLM_INT8 ? p.grp / 16 : 1;
        gemv_split_kernel<WD><<<(units * parts + kGemvWarps - 1) / kGemvWarps, kGemvThreads, smem, st>>>(pt, parts, (cpg & (cpg - 1)) == 0 ? __builtin_ctz(cpg) : -1);
        g_launches++;
        SLLM_LAUNCH_CHECK();
        return SLLM_OK;
    }
    const int grid = gemv_grid(units, 2);
    gemv_plain_kernel<WD><<<grid, kGemvThreads, smem, st>>>(pt);
    g_launches++;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}

int check_gemv_args(const void* W, int w_dtype, const float* scales, int group, int rows, int cols) {
    SLLM_REQUIRE(W && rows > 0 && cols > 0, SLLM_EINVAL, "gemv: null weight or empty shape");
    SLLM_REQUIRE(((uintptr_t)W & 15) == 0, SLLM_EINVAL, "gemv: weight pointer must be 16-byte aligned");
    const int E = w_dtype == SLLM_F32 ? 4 : w_dtype == SLLM_BF16 ? 8 : w_dtype == SLLM_INT8 ? 16 : 0;
    SLLM_REQUIRE(E != 0, SLLM_EINVAL, "gemv: unknown weight dtype %d", w_dtype);
    SLLM_REQUIRE(cols % E == 0, SLLM_ENOTSUP, "gemv: cols=%d must be a multiple of %d for this weight type", cols, E);
    if (w_dtype == SLLM_INT8)
        SLLM_REQUIRE(scales && group >= 16 && group % 16 == 0 && cols % group == 0, SLLM_EINVAL,
                     "gemv: int8 needs scales, group %% 16 == 0 and cols %% group == 0 (cols=%d group=%d)", cols, group);
    return SLLM_OK;
}

}  // namespace sllm

using namespace sllm;

extern "C" int sllm_gemv(const float* x, const void* W, int32_t w_dtype, const float* scales, int32_t group, float* y,
                         int32_t rows, int32_t cols, float scale, sllm_stream_t stream) {
    SLLM_REQUIRE(x && y, SLLM_EINVAL, "gemv: null vector");
    SLLM_REQUIRE(((uintptr_t)x & 15) == 0, SLLM_EINVAL, "gemv: x must be 16-byte aligned");
    if (int rc = check_gemv_args(W, w_dtype, scales, group, rows, cols)) return rc;
    PlainPolicy p{x, W, scales, y, group, rows, cols, scale};
    switch (w_dtype) {
        case SLLM_F32: return launch_plain<SLLM_F32>(p, as_stream(stream));
        case SLLM_BF16: return launch_plain<SLLM_BF16>(p, as_stream(stream));
        default: return launch_plain<SLLM_INT8>(p, as_stream(stream));
    }
}
