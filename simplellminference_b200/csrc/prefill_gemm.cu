// csrc/prefill_gemm.cu — the prefill GEMM on the 5th-generation tensor cores (sm_100a only).
//
//   C[T][N] = A[T][K] . W[N][K]^T      A = bf16 activations, W = bf16 weights, C = fp32 accumulators in TMEM
//
// One persistent CTA per SM, 192 threads, three roles (no role ever blocks another with __syncthreads):
//   warp 0 (one lane)  TMA producer: cp.async.bulk.tensor of a 128 x 64 A box and this CTA's W box per k-block into a ring of
//                      128B-swizzled stages, completion counted on the stage's "full" mbarrier;
//   warp 1 (one lane)  MMA issuer: 4 x tcgen05.mma.kind::f16 (K = 16 each) per stage, both operands through shared-memory
//                      descriptors; tcgen05.commit frees the stage / publishes the accumulator;
//   warps 2-5          epilogue: tcgen05.ld 32 columns at a time (one accumulator row per thread), fused epilogue
//                      (RoPE + KV-cache write, sigmoid(gate)*up, residual add), while the issuer already fills the
//                      second accumulator (TMEM holds two of up to 256 columns).
// Two cluster shapes: one SM per 128 x BN tile (cta_group::1, prompts of <= 128 rows and the T = 1 classifier), or the two SMs of
// a TPC on one 256 x BN tile (cta_group::2: each CTA stages its own 128 rows of A and BN/2 rows of W, the leader issues the MMAs,
// its commits are multicast to both CTAs). BN is a run-time multiple of 32; the residual-epilogue GEMMs may split K (pf_plan).
// W is read straight from the megakernel's TILED decode layout (megakernel.cuh) through a 4-D tensor map
// {k inside a K slice, row inside a tile, K slice, tile row}: prefill and decode share one copy of the weights.
// Rows of the tiled layout are in unit order, so the two values an epilogue needs together (RoPE partners,
// (up, gate)) sit in ADJACENT accumulator columns of the same thread.
// Bound: the tensor pipe inside a tile (a 256 x 224 tile's k-block of 64 takes 461 clocks of the 448 its products need), beside that some 2 us until the first operands are there and
// 4 us for the last tile's rows. What it took, measured back to back on matrices larger than L2 in turn, before | after: issuing loops without divisions (560 | 290 clocks per
// k-block), rows written by whole lines (a k-block beside an epilogue 2400 | 600 clocks), and an epilogue without a loop that indexes the accumulator registers, which had put them
// into local memory (1600 | 900 clocks per 32 columns). 2048 x 12288 x 4096: 186 | 143 us; 512 x 12288 x 4096: 65 | 46; 512 x 4096 x 4096: 31 | 20; 512 x 4096 x 11008: 64 | 41;
// 2048 x 6176 x 2048: 66 | 43; 2048 x 2048 x 2048: 26 | 19. L2 prefetch and stream-K were measured and dropped, and so was asking for the next k-block's barrier in advance.
#include <map>
#include <tuple>

#include "prefill.cuh"
#include "tcgen05.cuh"

namespace sllm {

extern int g_tune_pf_bn, g_tune_pf_pair, g_tune_pf_pdl, g_tune_pf_ksplit;
constexpr int kPfBM = 128, kPfBK = 64, kPfThreads = 192;
constexpr uint32_t kPfABytes = kPfBM * kPfBK * 2;
// PAIR = true: two CTAs of a cluster (the two SMs of a TPC) work on ONE 256 x BN tile with tcgen05.mma.cta_group::2 — each
// CTA stages its own 128 rows of A and its own BN/2 rows of W, so shared-memory traffic (TMA writes + tensor-core reads) and
// L2->SM traffic per flop are 2/3 of the single-CTA 128 x BN tile's.
// The N extent of a tile (BN) is a RUN-TIME multiple of 32 up to 256 (one tcgen05.mma takes any N that is a multiple of 16):
// the host picks the BN that fills the last wave best, e.g. 192 instead of 256 for a 512 x 12288 output on 74 SM pairs.
constexpr int kPfMaxStages = 12;
constexpr uint32_t kPfRingBytes = 192 * 1024;          // operand ring; stages = ring / (A box + this CTA's W box)
constexpr uint32_t kPfTmemCols = 512;                  // two accumulators of up to 256 fp32 columns
constexpr size_t kPfSmem = 1024 /*alignment slack*/ + kPfRingBytes + 512 /*barriers + tmem slot*/ + 4 * 4096 /*rows on their way through the epilogue*/;

struct PfDev {           // kernel-side view of PfGemmArgs
    int32_t T, N, m_tiles, n_tiles, BN;
    int32_t ksplit;       // > 1 (residual / accumulate epilogues only): a tile's k-blocks are cut into ksplit work units whose partial sums are ADDED to
                          // the residual stream with red.global.add — fills the machine when a GEMM has fewer tiles than SM pairs
    int32_t nkb, kb_per_seg, seg_elems, R, tiled;
    int32_t epilogue;
    int32_t a_rows;       // rows of A one CTA stages per k-block: 128, or (one-SM kernel, T < 128) T rounded up to the 8-row swizzle period —
                          // the rest of the 128-row operand tile is never loaded (its accumulator rows are never stored)
    float* out; int32_t ld_out, n_valid, vec_out;   // vec_out: rows of out may be written 16 bytes at a time
    uint16_t* q_out; uint8_t *kc, *vc; int32_t kv_dtype, q_loc, kv_loc, hd, S, pos0;
    const float *sin_t, *cos_t;
    uint16_t* s_out; int32_t I_loc;
    const float* bias;
    const int32_t* rows_dev;   // the row tiles beyond ceil(*rows_dev / tile rows) are skipped by every role alike
    int32_t groups;            // matrices one behind the other, each with its own count in rows_dev; T and N are then those of one group
    int32_t* status;           // where a wait that was given up is reported
    long long wait_clocks;     // and after how long it is
};

// Bounded wait on a barrier: false once `limit` clocks have passed or another thread of the CTA has given up. The kernel then tears down without its result and says
// so in the library's status word. (By the clock and not by polls: a poll may sleep.)
// Of a pair, the other CTA is told at once: what is on its way for one may reach into the other's memory, so both take their time before they leave.
__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t mapa_u32(const void* local, uint32_t cta) {   // shared::cluster address of `local` in CTA `cta`
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(s_addr(local)), "r"(cta));
    return r;
}
template <bool PAIR>
__device__ __forceinline__ bool pf_wait(uint64_t* bar, uint32_t parity, volatile int* gave_up, long long limit) {
    uint32_t done;
    long long since = 0;
    while (true) {
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(s_addr(bar)), "r"(parity) : "memory");
        if (done) return true;
        const long long now = clock64();
        if (!since) since = now;
        if (*gave_up || now - since > limit) break;
    }
    *gave_up = 1;
    if (PAIR) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa_u32(const_cast<const int*>(gave_up), cluster_ctarank() ^ 1)), "r"(1) : "memory");
    return false;
}

// ------------------------------------------------------------------------------------------ PTX -------
// PAIR: the cta_group::2 forms. The destination is this CTA's shared memory, the mbarrier may live in the peer CTA (shared::cluster address)
template <bool PAIR>
__device__ __forceinline__ void pf_load_2d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
    if constexpr (PAIR)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void pf_load_4d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, int c2, int c3, uint32_t bar) {
    if constexpr (PAIR)
        asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                     ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                     ::"r"(dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void mb_arrive_cluster(uint32_t bar_cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_alloc_pair(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(slot)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrives on the barrier at this offset in BOTH CTAs of the pair once all MMAs issued so far have completed
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(s_addr(bar)), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void tc_mma_bf16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) { return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16); }

// ------------------------------------------------------------------------------- fused epilogues ------
// All lanes of an epilogue warp call them together. v[0..31] = accumulator columns n0 .. n0+31 (n0 is a multiple of 32) of this lane's token row; `valid`: there is such a token.
// A store of 16 bytes into each of 32 rows reaches the L2 as 32 half sectors, and while they were written that way the operands of the next tile waited behind them: a
// k-block took 2400 clocks beside an epilogue and 580 without one. So rows change lanes first and whole lines (fp32) or sectors (bf16) are written.

// fp32 rows: through `tr`, 4 KB of shared memory of this warp (16-byte pieces of a row in the XOR swizzle); eight lanes then write the 128 bytes of one row
template <int MODE>      // 0 = store, 1 = add to what is there, 2 = reduction in L2 (no return value): for the partial sums of a split K
__device__ __forceinline__ void epi_rows(const PfDev& p, uint32_t tr, int t0, int t_limit, int t_shift, int n0, const uint32_t* v, bool bias) {
    const int lane = threadIdx.x & 31, sub = lane >> 3, c = lane & 7;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tr + lane * 128 + ((i ^ c) << 4)), "r"(v[4 * i]), "r"(v[4 * i + 1]), "r"(v[4 * i + 2]), "r"(v[4 * i + 3]) : "memory");
    __syncwarp();
    const int n = n0 + 4 * c;
    float4 x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int row = 4 * r + sub;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[r].x), "=f"(x[r].y), "=f"(x[r].z), "=f"(x[r].w) : "r"(tr + row * 128 + ((c ^ (row & 7)) << 4)) : "memory");
    }
    __syncwarp();
    if (bias) {
        const float4 b = make_float4(n < p.n_valid ? p.bias[n] : 0.f, n + 1 < p.n_valid ? p.bias[n + 1] : 0.f, n + 2 < p.n_valid ? p.bias[n + 2] : 0.f, n + 3 < p.n_valid ? p.bias[n + 3] : 0.f);
#pragma unroll
        for (int r = 0; r < 8; ++r) x[r] = make_float4(x[r].x + b.x, x[r].y + b.y, x[r].z + b.z, x[r].w + b.w);
    }
    float* dst = p.out + (size_t)(t0 + t_shift + sub) * p.ld_out + n;
    const size_t step = 4 * (size_t)p.ld_out;
    if (p.vec_out && n0 + 32 <= p.n_valid) {
        if (MODE == 1) {                                   // residual + projection (add_kernel.cpp:10-13)
            float4 y[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (t0 + 4 * r + sub < t_limit) y[r] = *reinterpret_cast<const float4*>(dst + r * step);
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = make_float4(y[r].x + x[r].x, y[r].y + x[r].y, y[r].z + x[r].z, y[r].w + x[r].w);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (t0 + 4 * r + sub >= t_limit) break;
            if (MODE == 2)
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + r * step), "f"(x[r].x), "f"(x[r].y), "f"(x[r].z), "f"(x[r].w) : "memory");
            else
                *reinterpret_cast<float4*>(dst + r * step) = x[r];
        }
    } else {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (t0 + 4 * r + sub >= t_limit) break;
            const float e[4] = {x[r].x, x[r].y, x[r].z, x[r].w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n + i < p.n_valid) {
                    if (MODE == 2) atomicAdd(dst + r * step + i, e[i]);
                    else dst[r * step + i] = MODE == 1 ? dst[r * step + i] + e[i] : e[i];
                }
        }
    }
}

// 32 bytes of every lane's own row at `own` (16-byte aligned; the neighbour's row lies `stride` bytes further for even lanes, before it for odd ones): a pair of lanes
// writes the even lane's row first, then the odd one's, 32 bytes each time
__device__ __forceinline__ void put_pair(uint8_t* own, ptrdiff_t stride, const uint4& a, const uint4& b, bool valid, bool peer_valid) {
    const bool odd = threadIdx.x & 1;
    uint4 s = odd ? a : b;
    s.x = __shfl_xor_sync(0xffffffffu, s.x, 1);
    s.y = __shfl_xor_sync(0xffffffffu, s.y, 1);
    s.z = __shfl_xor_sync(0xffffffffu, s.z, 1);
    s.w = __shfl_xor_sync(0xffffffffu, s.w, 1);
    uint8_t* even_row = odd ? own - stride + 16 : own;
    if (odd ? peer_valid : valid) *reinterpret_cast<uint4*>(even_row) = odd ? s : a;
    if (odd ? valid : peer_valid) *reinterpret_cast<uint4*>(even_row + stride) = odd ? b : s;
}
__device__ __forceinline__ uint4 pack_bf16x8(const float* x) { return make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7])); }

__device__ __forceinline__ void epi_gateup(const PfDev& p, int t, int n0, const uint32_t* v, bool valid, bool peer_valid) {
    const int u0 = n0 >> 1;
    float s[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float up = __uint_as_float(v[2 * i]), gate = __uint_as_float(v[2 * i + 1]);
        s[i] = (1.0f / (1.0f + expf(-gate))) * up;   // swiglu_kernel.cpp:12-13
    }
    uint16_t* dst = p.s_out + (size_t)t * p.I_loc + u0;
    if (u0 + 16 <= p.I_loc && (p.I_loc & 7) == 0) {
        put_pair(reinterpret_cast<uint8_t*>(dst), 2 * (ptrdiff_t)p.I_loc, pack_bf16x8(s), pack_bf16x8(s + 8), valid, peer_valid);
    } else if (valid) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (u0 + i < p.I_loc) dst[i] = f32_to_bf16_bits(s[i]);
    }
}

// 16 consecutive elements of a cache row per lane; the neighbour's row is the next position
__device__ __forceinline__ void kv_store16(uint8_t* cache, const PfDev& p, size_t elem, const float* x, bool valid, bool peer_valid) {
    if (p.kv_dtype == SLLM_BF16) {
        put_pair(cache + elem * 2, 2 * (ptrdiff_t)p.hd, pack_bf16x8(x), pack_bf16x8(x + 8), valid, peer_valid);
    } else {
        const uint4* q = reinterpret_cast<const uint4*>(x);
        put_pair(cache + elem * 4, 4 * (ptrdiff_t)p.hd, q[0], q[1], valid, peer_valid);
        put_pair(cache + elem * 4 + 32, 4 * (ptrdiff_t)p.hd, q[2], q[3], valid, peer_valid);
    }
}
__device__ __forceinline__ void kv_store1(uint8_t* cache, int kv_dtype, size_t elem, float x) {
    if (kv_dtype == SLLM_BF16) reinterpret_cast<uint16_t*>(cache)[elem] = f32_to_bf16_bits(x);
    else reinterpret_cast<float*>(cache)[elem] = x;
}

__device__ __forceinline__ void epi_qkv(const PfDev& p, int t, int n0, const uint32_t* v, bool valid, bool peer_valid) {
    const int half = p.hd >> 1, rope_units = (p.q_loc + p.kv_loc) >> 1, nunits = (p.q_loc + 2 * p.kv_loc) >> 1;
    const int u0 = n0 >> 1;
    const int pos = p.pos0 + t;
    if (u0 >= nunits) return;
    if ((half & 15) == 0 && u0 + 16 <= nunits) {
        // 16 units = 16 consecutive j of ONE head (half is a multiple of 16) or 32 consecutive V elements
        if (u0 < rope_units) {
            const int head = u0 / half, j0 = u0 - head * half;
            const size_t at = (size_t)(valid ? pos : p.pos0) * half + j0;
            const float4* sp = reinterpret_cast<const float4*>(p.sin_t + at);
            const float4* cp = reinterpret_cast<const float4*>(p.cos_t + at);
            alignas(16) float lo[16], hi[16];
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                const float4 s4 = sp[i4], c4 = cp[i4];
                const float ss[4] = {s4.x, s4.y, s4.z, s4.w}, cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = 4 * i4 + k;
                    const float a = __uint_as_float(v[2 * i]), b = __uint_as_float(v[2 * i + 1]);
                    lo[i] = a * cc[k] - b * ss[k];   // rope_kernel.cpp:36-37
                    hi[i] = b * cc[k] + a * ss[k];
                }
            }
            const int r0 = head * p.hd + j0;
            if (r0 < p.q_loc) {
                uint8_t* q = reinterpret_cast<uint8_t*>(p.q_out + (size_t)t * p.q_loc + r0);
                put_pair(q, 2 * (ptrdiff_t)p.q_loc, pack_bf16x8(lo), pack_bf16x8(lo + 8), valid, peer_valid);
                put_pair(q + 2 * half, 2 * (ptrdiff_t)p.q_loc, pack_bf16x8(hi), pack_bf16x8(hi + 8), valid, peer_valid);
            } else {
                const int kvh = (r0 - p.q_loc) / p.hd;
                const size_t e0 = ((size_t)kvh * p.S + pos) * p.hd + j0;
                kv_store16(p.kc, p, e0, lo, valid, peer_valid);
                kv_store16(p.kc, p, e0 + half, hi, valid, peer_valid);
            }
        } else {
            const int b2 = 2 * (u0 - rope_units);
            const int kvh = b2 / p.hd, j = b2 - kvh * p.hd;
            const size_t e0 = ((size_t)kvh * p.S + pos) * p.hd + j;
            alignas(16) float x[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(v[i]);
            kv_store16(p.vc, p, e0, x, valid, peer_valid);
            kv_store16(p.vc, p, e0 + 16, x + 16, valid, peer_valid);
        }
        return;
    }
    if (!valid) return;
#pragma unroll                       // (a loop that indexes v would put it into local memory)
    for (int i = 0; i < 16; ++i) {   // generic shapes: unit by unit
        const int u = u0 + i;
        if (u >= nunits) continue;
        const float a = __uint_as_float(v[2 * i]), b = __uint_as_float(v[2 * i + 1]);
        if (u < rope_units) {
            const int head = u / half, j = u - head * half;
            const float s = p.sin_t[(size_t)pos * half + j], c = p.cos_t[(size_t)pos * half + j];
            const float o0 = a * c - b * s, o1 = b * c + a * s;
            const int r0 = head * p.hd + j;
            if (r0 < p.q_loc) {
                p.q_out[(size_t)t * p.q_loc + r0] = f32_to_bf16_bits(o0);
                p.q_out[(size_t)t * p.q_loc + r0 + half] = f32_to_bf16_bits(o1);
            } else {
                const int kvh = (r0 - p.q_loc) / p.hd;
                const size_t e0 = ((size_t)kvh * p.S + pos) * p.hd + j;
                kv_store1(p.kc, p.kv_dtype, e0, o0);
                kv_store1(p.kc, p.kv_dtype, e0 + half, o1);
            }
        } else {
            const int b2 = 2 * (u - rope_units);
            const int kvh = b2 / p.hd, j = b2 - kvh * p.hd;
            const size_t e0 = ((size_t)kvh * p.S + pos) * p.hd + j;
            kv_store1(p.vc, p.kv_dtype, e0, a);
            kv_store1(p.vc, p.kv_dtype, e0 + 1, b);
        }
    }
}

// ------------------------------------------------------------------------------------------ kernel ----
template <bool PAIR>
__global__ void __launch_bounds__(kPfThreads, 1) pf_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                                                                const PfDev p) {
    constexpr int BM = PAIR ? 2 * kPfBM : kPfBM;          // rows of the (pair's) tile
    const int BN = p.BN;
    const int b_rows = PAIR ? BN / 2 : BN;                 // W rows staged by one CTA
    const uint32_t b_bytes = (uint32_t)b_rows * kPfBK * 2, stage_bytes = kPfABytes + b_bytes;
    const uint32_t tx_bytes = (uint32_t)p.a_rows * kPfBK * 2 + b_bytes;   // bytes the TMA really delivers per stage (a_rows < 128: skinny A)
    const int ST = min((int)(kPfRingBytes / stage_bytes), kPfMaxStages);
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;   // 0 = leader: issues the MMAs of the pair
    const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, nworkers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    extern __shared__ uint8_t pf_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pf_smem_raw) + 1023) & ~(uintptr_t)1023);   // SW128 tiles: 1024-byte aligned
    uint8_t* sA = smem;                                    // [ST] 128 x 64 bf16, 16 KB each
    uint8_t* sB = smem + (size_t)ST * kPfABytes;           // [ST] b_rows x 64 bf16 (multiples of 1024 bytes: b_rows % 8 == 0)
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPfRingBytes);
    uint64_t* empty = full + kPfMaxStages;
    uint64_t* tfull = empty + kPfMaxStages;     // [2] accumulator ready for the epilogue
    uint64_t* tempty = tfull + 2;     // [2] accumulator drained
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < ST; ++s) { mb_init(full + s, 1); mb_init(empty + s, 1); }
        for (int a = 0; a < 2; ++a) { mb_init(tfull + a, 1); mb_init(tempty + a, PAIR ? 8 : 4); }
        *gave_up = p.wait_clocks == 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // The forms of tcgen05.alloc and tcgen05.dealloc for a pair act on both CTAs' tensor memory: whoever issues one has to make sure that the peer runs already and is still there. Hence the barrier
    // of the pair in front of the first and the one behind the last (see the end). No third one is needed for the peer's allocation: the leader's first product waits for the peer's bytes, which
    // the peer asks for when it has its columns.
    if (PAIR) cluster_sync_all();   // and the peer's barriers are initialised before anything signals them
    if (warp == 1) { if (PAIR) tc_alloc_pair(tmem_slot, kPfTmemCols); else tc_alloc(tmem_slot, kPfTmemCols); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // programmatic dependent launch: everything above overlapped the previous kernel's tail; its results (A, the residual
    // stream) are visible after the wait. The next kernel may start ITS set-up as soon as every CTA here is past this point.
    pdl_wait();
    pdl_launch_dependents();
    // row counts left by an earlier kernel (tokens routed to an expert): every thread reads the same numbers, so the three roles walk the
    // same work units (all of group 0, then all of group 1, ...); with no rows at all the kernel only tears down
    struct Walk {
        const PfDev& p;
        int g, base, m_tiles;                             // group at hand, its first work unit, its row tiles
        __device__ __forceinline__ int tiles() const {
            return p.rows_dev ? min(p.m_tiles, (p.rows_dev[g] + BM - 1) / BM) : p.m_tiles;
        }
        __device__ __forceinline__ explicit Walk(const PfDev& q) : p(q), g(0), base(0) { m_tiles = tiles(); }
        __device__ __forceinline__ bool reach(int unit) {  // units come in ascending order
            while (unit - base >= m_tiles * p.n_tiles * p.ksplit) {
                base += m_tiles * p.n_tiles * p.ksplit;
                if (++g >= p.groups) return false;
                m_tiles = tiles();
            }
            return true;
        }
    };
    Walk walk(p);
    const bool gone = p.wait_clocks == 0;      // no wait is allowed at all: every role gives up in front of its first one (asked once and not by every wait: a k-block's 290 clocks)

    // One elected lane of either issuing warp runs its loop, with nothing in it that need not be: with an integer division and addresses made anew for every k-block either warp
    // took 560 clocks for one, whatever its width (a 256 x 256 tile's products need 512, a 256 x 128 tile's 256); like this some 290. The lane waits by itself: a lane that
    // only looked on could miss a phase while the elected one goes on.
    if (warp == 0) {
        if (elect_one()) {     // ===== TMA producer =====
            const uint32_t full_at = PAIR ? mapa_u32(full, 0) : s_addr(full), a_at = s_addr(sA), b_at = s_addr(sB);   // pair: both CTAs' bytes are counted on the LEADER's barriers
            int stage = 0;
            uint32_t phase = 0;
            bool ok = !gone;
            for (int unit = worker; ok && walk.reach(unit); unit += nworkers) {
                const int tile = (unit - walk.base) / p.ksplit, part = (unit - walk.base) - tile * p.ksplit;
                const int kb0 = (p.nkb * part) / p.ksplit, kb1 = (p.nkb * (part + 1)) / p.ksplit;
                const int m_tile = tile % walk.m_tiles, n_tile = tile / walk.m_tiles;   // consecutive workers share the weight tile (L2)
                const int row0 = walk.g * p.T + m_tile * BM + (int)rank * kPfBM;   // this CTA's 128 rows of A
                const int n0 = walk.g * p.N + n_tile * BN + (int)rank * b_rows;    // this CTA's rows of W
                const int w_row = p.tiled ? 0 : n0, w_tile = p.tiled ? n0 / p.R : 0;
                int ks = kb0 / p.kb_per_seg, kk = kb0 - ks * p.kb_per_seg;
                for (int kb = kb0; kb < kb1; ++kb) {
                    ok = pf_wait<PAIR>(empty + stage, phase ^ 1, gave_up, p.wait_clocks);
                    if (!ok) break;
                    const uint32_t bar = full_at + 8 * stage;
                    if (!PAIR) mb_expect(full + stage, tx_bytes);
                    else if (rank == 0) mb_expect(full + stage, 2 * tx_bytes);
                    pf_load_2d<PAIR>(a_at + (uint32_t)stage * kPfABytes, &tmA, ks * p.seg_elems + kk * kPfBK, row0, bar);
                    pf_load_4d<PAIR>(b_at + (uint32_t)stage * b_bytes, &tmB, kk * kPfBK, w_row, ks, w_tile, bar);
                    if (++kk == p.kb_per_seg) { kk = 0; ++ks; }
                    if (++stage == ST) { stage = 0; phase ^= 1; }
                }
            }
            // The last arrivals on `empty`, which no load waits for, come from the leader's SM: this CTA stays until they are in, its shared memory is another's afterwards. (A stage never
            // used is empty from the start.) They are in before the last accumulator is, so nothing waits longer for it.
            if (PAIR) {
#pragma unroll 1
                for (int s = 0; ok && s < ST; ++s) {
                    ok = pf_wait<PAIR>(empty + stage, phase ^ 1, gave_up, p.wait_clocks);
                    if (++stage == ST) { stage = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {   // ===== MMA issuer (pair: the leader CTA only) =====
            const uint32_t idesc = umma_idesc_bf16(BM, BN);
            const uint64_t a_desc = umma_desc_sw128(sA), b_desc = umma_desc_sw128(sB);
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = !gone;
            for (int unit = worker; ok && walk.reach(unit); unit += nworkers) {
                const int part = (unit - walk.base) % p.ksplit;
                const int n_kb = (p.nkb * (part + 1)) / p.ksplit - (p.nkb * part) / p.ksplit;
                ok = pf_wait<PAIR>(tempty + acc, acc_phase ^ 1, gave_up, p.wait_clocks);   // the epilogue has drained this accumulator
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * 256);
                for (int kb = 0; kb < n_kb; ++kb) {
                    ok = pf_wait<PAIR>(full + stage, phase, gave_up, p.wait_clocks);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t ad = a_desc + (uint64_t)((uint32_t)stage * (kPfABytes >> 4)), bd = b_desc + (uint64_t)((uint32_t)stage * (b_bytes >> 4));
#pragma unroll
                    for (int k = 0; k < kPfBK / 16; ++k) {   // +32 bytes along K inside the 128-byte swizzle atom = +2 in the address field
                        if (PAIR) tc_mma_bf16_pair(d_tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc, (kb | k) != 0);
                        else tc_mma_bf16(d_tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc, (kb | k) != 0);
                    }
                    if (PAIR) tc_commit_pair(empty + stage); else tc_commit(empty + stage);   // stage reusable once these MMAs have read it
                    if (++stage == ST) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                if (PAIR) tc_commit_pair(tfull + acc); else tc_commit(tfull + acc);           // accumulator complete
                if (++acc == 2) { acc = 0; acc_phase ^= 1; }
            }
        }
        __syncwarp();
    } else {               // ===== epilogue warps 2..5: TMEM lane quadrant = warp % 4 =====
        const int quad = warp & 3;
        const uint32_t tr = s_addr(smem + kPfRingBytes + 512 + quad * 4096);
        int acc = 0;
        uint32_t acc_phase = 0;
        const uint32_t tempty_leader[2] = {PAIR ? mapa_u32(tempty, 0) : 0u, PAIR ? mapa_u32(tempty + 1, 0) : 0u};
        for (int unit = worker; !gone && walk.reach(unit); unit += nworkers) {
            const int tile = (unit - walk.base) / p.ksplit;
            const int m_tile = tile % walk.m_tiles, n_tile = tile / walk.m_tiles;
            const int t0 = m_tile * BM + (int)rank * kPfBM + quad * 32, t = t0 + lane;
            const bool bias = p.bias && (unit - walk.base) % p.ksplit == 0;   // the bias rides on the first share of K
            // the warp goes on as one: what follows are instructions of all its lanes
            if (!__all_sync(0xffffffffu, pf_wait<PAIR>(tfull + acc, acc_phase, gave_up, p.wait_clocks))) break;
            tc_fence_after();
            const uint32_t src = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * 256);
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t v[32];
                __syncwarp();
                tc_ld32(src + (uint32_t)c0, v);
                if (c0 + 32 >= BN) {                     // the accumulator has been read: the next tile may have it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) { if (PAIR) mb_arrive_cluster(tempty_leader[acc]); else mb_arrive(tempty + acc); }
                }
                const int n0 = n_tile * BN + c0;
                if (t0 < p.T && n0 < p.N) {
                    if (p.epilogue == PF_EPI_QKV) epi_qkv(p, t, n0, v, t < p.T, (t ^ 1) < p.T);
                    else if (p.epilogue == PF_EPI_GATEUP) epi_gateup(p, t, n0, v, t < p.T, (t ^ 1) < p.T);
                    else if (p.ksplit > 1) epi_rows<2>(p, tr, t0, p.T, walk.g * p.T, n0, v, bias);
                    else if (p.epilogue == PF_EPI_RESID) epi_rows<1>(p, tr, t0, p.T, walk.g * p.T, n0, v, bias);
                    else epi_rows<0>(p, tr, t0, p.T, walk.g * p.T, n0, v, bias);
                }
            }
            if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        __syncwarp();
    }
    tc_fence_before();
    if (PAIR) cluster_sync_all(); else __syncthreads();   // pair: nobody leaves while the peer may still signal its barriers / read its operands
    if (*gave_up) tc_gave_up(p.status);                   // set, if at all, in front of the barrier
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) tc_dealloc_pair(tmem_base, kPfTmemCols); else tc_dealloc(tmem_base, kPfTmemCols);
    }
    // pair: nobody leaves before both have given up the tensor memory. An SM whose CTA had left could hold another kernel's CTA, with columns of its own, when the peer's dealloc for the pair came
    // through; the wait for columns is the one in this kernel that nothing bounds.
    if (PAIR) cluster_sync_all();
}

// -------------------------------------------------------------------------------------------- host ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

struct PfCache {
    std::map<std::tuple<const void*, int, int, int, int>, CUtensorMap> weights;   // (W, N, K, tiled, rows per box)
};
PfCache* pf_cache_create() { return new PfCache(); }
void pf_cache_destroy(PfCache* c) { delete c; }

int tc_encode_bf16(CUtensorMap* tm, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes, const cuuint32_t* box) {
    EncodeTiledFn fn = encode_fn();
    SLLM_REQUIRE(fn, SLLM_ESTATE, "cuTensorMapEncodeTiled is not available from this driver");
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    const CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides_bytes, box, ones,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    SLLM_REQUIRE(r == CUDA_SUCCESS, SLLM_EINVAL, "cuTensorMapEncodeTiled failed (%d): rank %d dims %llu %llu box %u %u", (int)r, rank,
                 (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1]);
    return SLLM_OK;
}

const char* pf_unsupported_reason(int w_dtype, int hd, int d, int q_loc, int I_loc) {
    if (w_dtype != SLLM_BF16) return "batched prefill needs bf16 weights (tensor-core operands)";
    if (hd != 64 && hd != 128) return "batched prefill attention is instantiated for head_dim 64 and 128";
    if (d % 8 || q_loc % 8 || I_loc % 8) return "row lengths must be multiples of 8 elements (16-byte TMA strides)";
    return nullptr;
}

template <bool PAIR>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const PfDev& p, cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        SLLM_CUDA(cudaFuncSetAttribute(pf_gemm_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPfSmem));
        configured = true;
    }
    const int workers = (int)std::min<long long>(PAIR ? sm_count() / 2 : sm_count(), (long long)p.m_tiles * p.n_tiles * p.ksplit * p.groups);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(PAIR ? 2 * workers : workers);
    cfg.blockDim = dim3(kPfThreads);
    cfg.dynamicSmemBytes = kPfSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = PAIR ? 2 : 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_tune_pf_pdl ? 2 : 1;
    SLLM_CUDA(cudaLaunchKernelEx(&cfg, pf_gemm_kernel<PAIR>, tmA, tmB, p));
    g_launches++;
    return SLLM_OK;
}

// Host-side plan of one GEMM: cluster shape, N extent of a tile, K split, k-blocks. Pure arithmetic (no device access beyond the
// cached SM count), exposed as sllm_prefill_gemm_plan for tests.
struct PfPlan { int pair, bn, ksplit, m_tiles, n_tiles, nkb, kb_per_seg, seg_elems, R; TileGeom g; };
static PfPlan pf_plan(int T, int N, int K, int tiled, int epilogue, int bn_forced, int groups = 1) {
    PfPlan pl{};
    // more than one 128-row block of tokens: two SMs share a 256-row tile (tcgen05 cta_group::2)
    pl.pair = g_tune_pf_pair >= 0 ? (g_tune_pf_pair != 0) : (T > kPfBM);
    const int BM = pl.pair ? 2 * kPfBM : kPfBM;
    pl.m_tiles = (T + BM - 1) / BM;
    if (tiled) {
        pl.g = mega_tile_geom(N, K, SLLM_BF16);
        pl.seg_elems = pl.g.SC * 8; pl.R = pl.g.R;
        pl.kb_per_seg = (pl.seg_elems + kPfBK - 1) / kPfBK;
        pl.nkb = pl.g.KS * pl.kb_per_seg;
    } else {
        pl.seg_elems = K; pl.R = 1;
        pl.kb_per_seg = (K + kPfBK - 1) / kPfBK;
        pl.nkb = pl.kb_per_seg;
    }
    // N extent of a tile (a multiple of 32 up to 256) and, for the residual epilogue, a split of K: a work unit is reckoned as k-blocks x operand rows per k-block plus the
    // epilogue of its tile, and the GEMM takes ceil(units / workers) waves of it; the cheapest combination is taken. The operand rows stand in for what a k-block takes, which is max(2 BN,
    // 290) clocks (measured, two SMs a tile): by those the choice is up to 6 % off, e.g. for 512 x 22016 x 4096 224 columns in three waves (86 016 clocks) where 160 in four take 81 920.
    int bn = bn_forced ? bn_forced : g_tune_pf_bn;
    int ksplit = 1;
    if (bn < 32 || bn > 256 || bn % 32) {
        const int workers = pl.pair ? sm_count() / 2 : sm_count();
        const bool adds = epilogue == PF_EPI_RESID || epilogue == PF_EPI_ACCUM;   // the epilogues whose partial sums may meet in L2
        const int max_split = (adds && g_tune_pf_ksplit != 0) ? (g_tune_pf_ksplit > 0 ? g_tune_pf_ksplit : 4) : 1;
        double best = 1e30;
        for (int b = 256; b >= 64; b -= 32) {
            for (int sp = 1; sp <= max_split; ++sp) {
                if (sp > 1 && pl.nkb / sp < 8) break;   // keep at least 8 k-blocks per work unit
                const long units = (long)pl.m_tiles * ((N + b - 1) / b) * sp * groups;
                const int a_rows = (!pl.pair && T < kPfBM) ? (T + 7) / 8 * 8 : kPfBM;   // operand rows a CTA really ingests per k-block
                const double unit_cost = (double)((pl.nkb + sp - 1) / sp) * (a_rows + (pl.pair ? b / 2 : b)) + 10.0 * b;
                const double c = (double)((units + workers - 1) / workers) * unit_cost;
                if (c < best - 1e-9) { best = c; bn = b; ksplit = sp; }
            }
        }
    } else if ((epilogue == PF_EPI_RESID || epilogue == PF_EPI_ACCUM) && g_tune_pf_ksplit > 0 && pl.nkb / g_tune_pf_ksplit >= 1) {
        ksplit = g_tune_pf_ksplit;
    }
    pl.bn = bn; pl.ksplit = ksplit;
    pl.n_tiles = (N + bn - 1) / bn;
    return pl;
}

int pf_gemm(PfCache* cache, const PfGemmArgs& a, cudaStream_t st) {
    SLLM_REQUIRE(cache && a.A && a.W && a.T > 0 && a.N > 0 && a.K > 0, SLLM_EINVAL, "pf_gemm: bad argument");
    SLLM_REQUIRE(a.K % 8 == 0, SLLM_ENOTSUP, "pf_gemm: K=%d must be a multiple of 8", a.K);
    const int groups = std::max(1, a.groups);
    SLLM_REQUIRE(groups == 1 || (!a.tiled && a.epilogue == PF_EPI_STORE && !a.bias && a.n_valid == a.N), SLLM_EINVAL, "pf_gemm: a grouped product only stores");
    PfPlan pl = pf_plan(groups > 1 && a.rows_hint > 0 ? std::min(a.rows_hint, a.T) : a.T, a.N, a.K, a.tiled, a.epilogue, a.bn, groups);
    if (groups > 1) pl.m_tiles = (a.T + (pl.pair ? 2 : 1) * kPfBM - 1) / ((pl.pair ? 2 : 1) * kPfBM);   // the most a group can hold
    const bool pair = pl.pair != 0;
    const int bn = pl.bn, ksplit = pl.ksplit;
    const TileGeom g = pl.g;
    PfDev p{};
    p.T = a.T; p.N = a.N; p.tiled = a.tiled; p.epilogue = a.epilogue;
    p.m_tiles = pl.m_tiles; p.seg_elems = pl.seg_elems; p.R = pl.R; p.kb_per_seg = pl.kb_per_seg; p.nkb = pl.nkb;
    p.ksplit = ksplit;
    p.BN = bn;
    p.n_tiles = pl.n_tiles;
    p.out = a.out; p.ld_out = a.ld_out; p.n_valid = a.n_valid;
    p.vec_out = a.ld_out % 4 == 0 && ((uintptr_t)a.out % 16) == 0;
    p.q_out = a.q_out; p.kc = a.k_cache; p.vc = a.v_cache; p.kv_dtype = a.kv_dtype; p.q_loc = a.q_loc; p.kv_loc = a.kv_loc; p.hd = a.hd; p.S = a.S;
    p.pos0 = a.pos0; p.sin_t = a.sin_t; p.cos_t = a.cos_t; p.s_out = a.s_out; p.I_loc = a.I_loc;
    p.bias = (a.epilogue == PF_EPI_STORE || a.epilogue == PF_EPI_RESID || a.epilogue == PF_EPI_ACCUM) ? a.bias : nullptr;
    p.rows_dev = a.rows_dev;
    p.groups = groups;
    if (int rc = status_check()) return rc;
    if (int rc = status_word(&p.status)) return rc;
    p.wait_clocks = kPollClocks * g_tune_tc_polls;

    CUtensorMap tmA;
    {
        const cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.T * groups};
        const cuuint64_t strides[1] = {(cuuint64_t)a.K * 2};
        p.a_rows = (!pair && a.T < kPfBM) ? (a.T + 7) / 8 * 8 : kPfBM;
        const cuuint32_t box[2] = {kPfBK, (cuuint32_t)p.a_rows};
        if (int rc = tc_encode_bf16(&tmA, a.A, 2, dims, strides, box)) return rc;
    }
    const int box_rows = pair ? bn / 2 : bn;   // W rows one CTA stages per k-block
    const auto key = std::make_tuple(a.W, a.N * groups, a.K, a.tiled, box_rows);
    auto it = cache->weights.find(key);
    if (it == cache->weights.end()) {
        CUtensorMap tmB;
        if (a.tiled) {
            const cuuint64_t dims[4] = {(cuuint64_t)p.seg_elems, (cuuint64_t)g.R, (cuuint64_t)g.KS, (cuuint64_t)g.ntr};
            const cuuint64_t strides[3] = {(cuuint64_t)g.SC * 16, (cuuint64_t)g.tile_bytes, (cuuint64_t)g.KS * g.tile_bytes};
            const cuuint32_t box[4] = {kPfBK, (cuuint32_t)g.R, 1, (cuuint32_t)(box_rows / g.R)};
            if (int rc = tc_encode_bf16(&tmB, a.W, 4, dims, strides, box)) return rc;
        } else {
            const cuuint64_t rows = (cuuint64_t)a.N * groups;
            const cuuint64_t dims[4] = {(cuuint64_t)a.K, rows, 1, 1};
            const cuuint64_t strides[3] = {(cuuint64_t)a.K * 2, (cuuint64_t)a.K * 2 * rows, (cuuint64_t)a.K * 2 * rows};
            const cuuint32_t box[4] = {kPfBK, (cuuint32_t)box_rows, 1, 1};
            if (int rc = tc_encode_bf16(&tmB, a.W, 4, dims, strides, box)) return rc;
        }
        it = cache->weights.emplace(key, tmB).first;
    }
    return pair ? launch<true>(tmA, it->second, p, st) : launch<false>(tmA, it->second, p, st);
}

}  // namespace sllm

extern "C" int sllm_prefill_gemm_bf16(const void* A, const void* W, float* C, int32_t T, int32_t N, int32_t K, int32_t bn, sllm_stream_t stream) {
    using namespace sllm;
    SLLM_REQUIRE(A && W && C, SLLM_EINVAL, "null argument");
    static PfCache* cache = pf_cache_create();
    cache->weights.clear();   // callers may reuse addresses for different matrices
    PfGemmArgs a{};
    a.A = A; a.W = W; a.T = T; a.N = N; a.K = K; a.tiled = 0; a.epilogue = PF_EPI_STORE; a.out = C; a.ld_out = N; a.n_valid = N; a.bn = bn;
    return pf_gemm(cache, a, as_stream(stream));
}

extern "C" int sllm_prefill_gemm_plan(int32_t T, int32_t N, int32_t K, int32_t residual_epilogue, int32_t* two_sm, int32_t* bn, int32_t* ksplit,
                                      int32_t* work_units) {
    using namespace sllm;
    SLLM_REQUIRE(T > 0 && N > 0 && K > 0 && K % 8 == 0, SLLM_EINVAL, "bad GEMM shape");
    const PfPlan pl = pf_plan(T, N, K, /*tiled=*/0, residual_epilogue ? PF_EPI_RESID : PF_EPI_STORE, 0);
    if (two_sm) *two_sm = pl.pair;
    if (bn) *bn = pl.bn;
    if (ksplit) *ksplit = pl.ksplit;
    if (work_units) *work_units = pl.m_tiles * pl.n_tiles * pl.ksplit;
    return SLLM_OK;
}
