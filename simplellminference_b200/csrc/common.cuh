// csrc/common.cuh — shared device/host helpers for libsllm_b200.so (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>

#include "../../include/sllm_b200.h"

namespace sllm {

// ------------------------------------------------------------------------------------- errors --------
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);

#define SLLM_CUDA(call)                                                      \
    do {                                                                     \
        cudaError_t _e = (call);                                             \
        if (_e != cudaSuccess) return ::sllm::cuda_fail(_e, #call, __FILE__, __LINE__); \
    } while (0)

#define SLLM_REQUIRE(cond, code, ...)      \
    do {                                   \
        if (!(cond)) {                     \
            ::sllm::set_error(__VA_ARGS__); \
            return (code);                 \
        }                                  \
    } while (0)

// What kernels have to report. A kernel that gives up a bounded wait stores kStatusWait in a word of mapped host memory, since it returns like any other;
// the library's next call that launches or waits returns SLLM_ETIMEOUT for it, once. kStatusBatch: index arrays on the device contradict the host's counts (SLLM_EINVAL).
constexpr int32_t kStatusWait = 1, kStatusBatch = 2;
extern int32_t* g_status;          // the word, nullptr until a kernel that may set it has been launched
int status_word(int32_t** word);   // makes it (also while a stream is being captured)
int status_take();                 // reports and clears
inline int status_check() { return g_status && *reinterpret_cast<volatile int32_t*>(g_status) ? status_take() : SLLM_OK; }

// Every launcher ends with this: a launch-configuration error surfaces here, not at the next sync.
#define SLLM_LAUNCH_CHECK()                              \
    do {                                                 \
        SLLM_CUDA(cudaGetLastError());                   \
        if (int _s = ::sllm::status_check()) return _s;  \
    } while (0)
// The same without the word: for a kernel that may set it, whose launcher has looked at it before (status_check), and for launches behind one in the same call, which would
// otherwise report this very call, or not, by how fast the kernel gives up.
#define SLLM_LAUNCH_CHECK_ONLY() SLLM_CUDA(cudaGetLastError())
// A wait of the library for a stream whose results it hands out.
#define SLLM_WAIT(stream)                                \
    do {                                                 \
        SLLM_CUDA(cudaStreamSynchronize(stream));        \
        if (int _s = ::sllm::status_check()) return _s;  \
    } while (0)

inline cudaStream_t as_stream(sllm_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

int sm_count();             // cached cudaDevAttrMultiProcessorCount of the current device
int smem_optin_bytes();     // cached cudaDevAttrMaxSharedMemoryPerBlockOptin
extern thread_local int64_t g_launches;   // launches issued by this thread (gpu_launches accounting)

// Launch attribute holder: programmatic dependent launch on/off (griddepcontrol in the kernels is a no-op
// when the attribute is absent).
struct LaunchCfg {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    LaunchCfg(dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl) {
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 1 : 0;
    }
};

// A kernel that calls after_previous() on every path: in a captured step it may become resident while the kernel before it still runs (sllm_graph_overlap). The
// launch itself is an ordinary one.
void overlap_kernel(const void* kernel, bool alone);
template <class F>
inline F* overlapping(F* kernel) {
    overlap_kernel(reinterpret_cast<const void*>(kernel), false);
    return kernel;
}
// The same, but early only where the launch is a single CTA: for kernels of few CTAs with much work each. Becoming resident while the kernel in front still holds most SMs, they
// end up several to an SM and take that much longer. Measured, us a step with the edge in front of them early | not: attention in latent heads (Vasosun, width 1024, four
// requests) 1017 | 927, a seam that convolves 1017 | 1003, experts' activation 1017 | 1005 (with one request, where those two are one CTA, 572 | 577 and 575), attention whose
// heads are mixed (Lovulix, width 1024, 64 requests) 1369 | 1092, rotation of latent queries (Sopetar, width 2048, 64) 1410 | 1397, products in tiles of 64 x 64 (Munazen, width
// 2048, 32) 14590 | 11400.
template <class F>
inline F* overlapping_alone(F* kernel) {
    overlap_kernel(reinterpret_cast<const void*>(kernel), true);
    return kernel;
}

// ------------------------------------------------------------------------------------- device --------
#ifdef __CUDACC__

constexpr int kWarp = 32;

// PDL: let the next kernel in the stream start its prologue / wait for the previous kernel's results.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// What a kernel launched through overlapping() does before it touches memory that another kernel writes or reads: every thread, on every path. It waits until the
// kernel in front has completed and then lets the one behind become resident. In that order: with the two exchanged a captured Nelutar step took 15 us longer (CTAs
// that only wait hold places which the step's other branches need). Data from other kernels are read without the read-only path (no __restrict__ in these
// kernels): those loads need not stay behind the wait.
// A launch of several waves does not signal: the one behind it could come in only with its last wave, and the signal costs 0.3 ns a CTA (a convolution over 2048 tokens of 1024
// channels, 16384 CTAs: 20.6 us with it, 16.5 like this, 15.3 without the instruction).
constexpr unsigned kSignalCtas = 8 * 148;
__device__ __forceinline__ void after_previous() {
    pdl_wait();
    if (gridDim.x * gridDim.y * gridDim.z <= kSignalCtas) pdl_launch_dependents();
}

// 128-bit streaming load of weights: read-only path, do not pollute L1 (each byte is used exactly once).
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}
// the same for data that the kernel in front may still have been writing when this one became resident (after_previous())
__device__ __forceinline__ uint4 ld_stream(const void* p) {
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ uint2 ldg_stream8(const void* p) {
    uint2 r;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// block-wide sum; `red` = shared scratch of >= 33 floats; every thread gets the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nw ? red[lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    float r = red[32];
    __syncthreads();
    return r;
}

// Index of the largest of n values (the first of equals), in thread 0 of a CTA of up to 1024 threads; NaN is never chosen, 0 if nothing is. Bound: what one SM reads; sixteen
// bytes a load and eight loads on their way per thread (one value a load took 10.8 us for 32000 values).
__device__ __forceinline__ void better_of(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
__device__ __forceinline__ int block_argmax(const float* x, int n, float* sv, int* si) {     // sv, si: 32 values of shared memory each
    float v = -INFINITY;
    int idx = 0x7fffffff;
    const int body = (reinterpret_cast<uintptr_t>(x) & 15) ? 0 : n / 4;
    constexpr int kAhead = 8;
    for (int c = threadIdx.x; c < body; c += kAhead * blockDim.x) {
        float4 q[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const int at = c + k * (int)blockDim.x;
            q[k] = at < body ? reinterpret_cast<const float4*>(x)[at] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const int at = c + k * (int)blockDim.x;
            if (at >= body) break;          // a value of -infinity may be the largest there is, but not one that stands in for nothing
            better_of(v, idx, q[k].x, 4 * at);
            better_of(v, idx, q[k].y, 4 * at + 1);
            better_of(v, idx, q[k].z, 4 * at + 2);
            better_of(v, idx, q[k].w, 4 * at + 3);
        }
    }
    for (int i = 4 * body + threadIdx.x; i < n; i += blockDim.x) better_of(v, idx, x[i], i);
    for (int o = 16; o > 0; o >>= 1) better_of(v, idx, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, idx, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sv[warp] = v; si[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        v = lane < nw ? sv[lane] : -INFINITY;
        idx = lane < nw ? si[lane] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) better_of(v, idx, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, idx, o));
    }
    return idx == 0x7fffffff ? 0 : idx;
}

// bf16 <-> fp32 by bit manipulation (RNE), identical to oracle/synth_weights.c:syn_round_bf16
__device__ __forceinline__ float bf16_lo(uint32_t packed) { return __uint_as_float(packed << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t packed) { return __uint_as_float(packed & 0xffff0000u); }
__device__ __forceinline__ uint16_t f32_to_bf16_bits(float x) {
    uint32_t u = __float_as_uint(x);
    if ((u & 0x7f800000u) != 0x7f800000u) u += 0x7fffu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}

#endif  // __CUDACC__

}  // namespace sllm
