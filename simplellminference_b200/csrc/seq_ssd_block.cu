// csrc/seq_ssd_block.cu — state-space duality (Mamba-2) over portions of prompts in blocks of 64 tokens on the tensor cores (bf16 mode). Per head, with G_i
// the running sum of the decays' logarithms inside a block and S0 [state][column] the state it starts from,
//     y_i = e^G_i S0^T C_i + sum_{j<=i} (C_i . B_j) e^(G_i - G_j) dt_j x_j + D x_i,        S' = e^G_n S0 + sum_j e^(G_n - G_j) dt_j B_j x_j^T
// (1) seq_ssd_prepare_kernel: what does not depend on the state, all blocks in parallel. B and C belong to a group of heads, so their tensor-core fragments
// and the products C_i . B_j (fp32) are made once per (block, group); step sizes and G once per (block, head).
// (2) seq_ssd_walk_kernel, CTA = (portion, head, 32 columns), 16 warps: S^T stays in the accumulators (fp32) from the portion's first token to its last,
// a warp owning 16 columns x an eighth of the states (and of the tokens); it is handed to the others as A fragments through shared memory once per block. Everything is
// computed transposed (columns are rows), so that accumulators become operands register for register. Every operand is three bf16 terms (24 bits), of whose
// products the six largest are kept, with fp32 sums (ssd_mma): the passes over ranges that this replaces for portions work on fp32 products, and the error
// must not grow. Decays are applied in fp32 to accumulators, to x before it is split and to the C_i . B_j, never to the shared fragments. No factor exceeds 1.
// Bound: 1776 mma per block and CTA (3600 clocks of an SM's tensor pipe) beside 85 KB of fragments from L2, which are fp32 and split where they are used (three
// terms would not fit twice). Error of the outputs alone against float64, ranges | blocks: 1.3e-7 | 1.3e-7 at usual decays, 1.7e-6 | 2.4e-7 at memories of
// thousands of tokens; two terms left 4.5e-6 and 6.1e-6. Measured, 2048 tokens, 64 heads of 64 columns, 128 states: ranges 698 us, blocks 193 us (with two terms 146:
// the walk 125, with 8 warps of twice the work 137). 2048 tokens of few heads are better off in ranges (8 heads 105 | 185 us).
#include "seq_attn.cuh"
#include "seq_ssd_block.cuh"

namespace sllm {

constexpr int kSsdCols = 32, kSsdThreads = 256, kSsdWalk = 512;      // columns of a walk's CTA, threads of the preparation, of the walk
constexpr float kSsdLog2e = 1.4426950408889634f;
constexpr int kSsdLdx = kSsdCols + 4;                         // padded row of x in shared memory

// fp32 fragments of a (block, group), four floats per lane: C as [token tile][k-step of states][lane], B as [state tile][k-step of tokens][lane], the
// products as [tile of i][k-step of j][lane] for the k-steps that hold a j <= i (ssd_w_tile)
template <int NK> struct SsdGroup {
    static constexpr int kC = 8 * (NK / 16) * 512, kB = (NK / 8) * 4 * 512, kW = 20 * 512, kBytes = kC + kB + kW;
};
__device__ __forceinline__ int ssd_w_tile(int nt, int ks) { return ((nt + 1) / 2) * ((nt + 2) / 2) + ks; }
static_assert(SsdGroup<128>::kBytes == ssd_block_group_bytes(128) && SsdGroup<64>::kBytes == ssd_block_group_bytes(64), "scratch sizes");

template <int NK>
__global__ void __launch_bounds__(kSsdThreads) seq_ssd_prepare_kernel(SsdBlockArgs p, int vec) {
    extern __shared__ __align__(16) float sp_sm[];
    const sllm_seq_batch& b = p.b;
    const size_t id = blockIdx.x;                            // this block's number in the scratch: whose is it?
    __shared__ int owner;
    if (threadIdx.x == 0) owner = -1;
    __syncthreads();
    for (int i = threadIdx.x; i < b.nseg; i += kSsdThreads) {
        const size_t first = ssd_block_id(b.seg_tile0[i], i, 0);
        if (id >= first && id < first + (b.seg_len[i] + kSsdBlock - 1) / kSsdBlock) owner = i;
    }
    __syncthreads();
    const int seg = owner;
    if (seg < 0) return;
    const int off = (int)(id - ssd_block_id(b.seg_tile0[seg], seg, 0)) * kSsdBlock, n = min(kSsdBlock, b.seg_len[seg] - off), start = b.seg_start[seg] + off;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.y >= p.groups) {                       // step sizes and running sums, a warp per head
        const int h = ((int)blockIdx.y - p.groups) * (kSsdThreads / 32) + warp;
        if (h >= p.heads) return;
        const float lg = -expf(p.A_log[h]) * kSsdLog2e, bias = p.dt_bias[h];
        float d0 = lane < n ? seq_softplus(p.step[(size_t)(start + lane) * p.lda + h] + bias) : 0.0f;
        float d1 = lane + 32 < n ? seq_softplus(p.step[(size_t)(start + lane + 32) * p.lda + h] + bias) : 0.0f;
        // A strong decay brings the sums to thousands while the differences that matter stay near zero: summed in double, kept as two fp32 terms
        double g0 = (double)(lg * d0), g1 = (double)(lg * d1);
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            const double u0 = __shfl_up_sync(0xffffffffu, g0, o), u1 = __shfl_up_sync(0xffffffffu, g1, o);
            if (lane >= o) {
                g0 += u0;
                g1 += u1;
            }
        }
        g1 += __shfl_sync(0xffffffffu, g0, 31);
        float* rec = p.head_ws + (id * p.heads + h) * (3 * kSsdBlock);
        rec[lane] = (float)g0;
        rec[lane + 32] = (float)g1;
        rec[kSsdBlock + lane] = (float)(g0 - (double)(float)g0);
        rec[kSsdBlock + lane + 32] = (float)(g1 - (double)(float)g1);
        rec[2 * kSsdBlock + lane] = d0;
        rec[2 * kSsdBlock + lane + 32] = d1;
        return;
    }
    constexpr int ld = NK + 4;
    float* s_b = sp_sm;
    float* s_c = s_b + kSsdBlock * ld;
    float (*s_w)[kSsdBlock + 1] = reinterpret_cast<float (*)[kSsdBlock + 1]>(s_c + kSsdBlock * ld);
    const int grp = blockIdx.y;
    for (int i = threadIdx.x; i < kSsdBlock * NK / 4; i += kSsdThreads) {
        const int tok = i / (NK / 4), st = (i % (NK / 4)) * 4;
        const size_t t = start + min(tok, n - 1);
        auto four = [&](const float* base, int ldr) {
            const float* row = base + t * ldr + (size_t)grp * p.n_state;
            if (tok >= n) return make_float4(0.f, 0.f, 0.f, 0.f);
            if (vec && st < p.n_state) return *reinterpret_cast<const float4*>(row + st);
            return make_float4(st < p.n_state ? row[st] : 0.f, st + 1 < p.n_state ? row[st + 1] : 0.f, st + 2 < p.n_state ? row[st + 2] : 0.f,
                               st + 3 < p.n_state ? row[st + 3] : 0.f);
        };
        *reinterpret_cast<float4*>(s_b + tok * ld + st) = four(p.B, p.ldb);
        *reinterpret_cast<float4*>(s_c + tok * ld + st) = four(p.C, p.ldc);
    }
    __syncthreads();
    {   // C . B^T, four by four per thread
        const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
        float acc[4][4] = {};
        for (int k0 = 0; k0 < NK; k0 += 16) {                // sums of 16 products, then the sum of those: fewer roundings in a row
            float part[4][4] = {};
#pragma unroll
            for (int k = k0; k < k0 + 16; k += 4) {
                float4 cv[4], bv[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    cv[r] = *reinterpret_cast<const float4*>(s_c + (ti + 16 * r) * ld + k);
                    bv[r] = *reinterpret_cast<const float4*>(s_b + (tj + 16 * r) * ld + k);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        part[i][j] = fmaf(cv[i].x, bv[j].x, fmaf(cv[i].y, bv[j].y, fmaf(cv[i].z, bv[j].z, fmaf(cv[i].w, bv[j].w, part[i][j]))));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s_w[ti + 16 * i][tj + 16 * j] = acc[i][j];
    }
    using Group = SsdGroup<NK>;
    uint8_t* rec = p.group_ws + (id * p.groups + grp) * Group::kBytes;
    for (int x = threadIdx.x; x < Group::kC / 16; x += kSsdThreads) {
        const int l = x & 31, g = l >> 2, c = l & 3, ks = (x >> 5) % (NK / 16), nt = (x >> 5) / (NK / 16);
        const float* row = s_c + (nt * 8 + g) * ld + ks * 16 + 2 * c;
        reinterpret_cast<float4*>(rec)[x] = make_float4(row[0], row[1], row[8], row[9]);
    }
    for (int x = threadIdx.x; x < Group::kB / 16; x += kSsdThreads) {
        const int l = x & 31, g = l >> 2, c = l & 3, ks = (x >> 5) & 3, nt = x >> 7;
        const float* at = s_b + (ks * 16 + 2 * c) * ld + nt * 8 + g;
        reinterpret_cast<float4*>(rec + Group::kC)[x] = make_float4(at[0], at[ld], at[8 * ld], at[9 * ld]);
    }
    __syncthreads();
    for (int x = threadIdx.x; x < 8 * 4 * 32; x += kSsdThreads) {
        const int l = x & 31, g = l >> 2, c = l & 3, ks = (x >> 5) & 3, nt = x >> 7;
        if (ks > nt / 2) continue;
        const float* row = &s_w[nt * 8 + g][ks * 16 + 2 * c];
        reinterpret_cast<float4*>(rec + Group::kC + Group::kB)[ssd_w_tile(nt, ks) * 32 + l] = make_float4(row[0], row[1], row[8], row[9]);
    }
}

__device__ __forceinline__ bool ssd_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// A k-step of a product at fp32 accuracy: both operands are three bf16 terms (24 bits), of whose products the six largest are kept (the rest is below 2^-24). The
// product of the first terms starts from zero and is added to `sum` with ordinary rounding, because the tensor core's own accumulation truncates; the
// others are 2^8 times smaller and share two accumulators.
struct SsdTerms { uint32_t h[4], m[4], l[4]; };
struct SsdSum { float s[4], d[2][4]; };
__device__ __forceinline__ void ssd_mma(SsdSum& y, const SsdTerms& a, const float4& f) {
    uint32_t h0, h1, m0, m1, l0, l1;
    split3_bf16(f.x, f.y, h0, m0, l0);
    split3_bf16(f.z, f.w, h1, m1, l1);
    float p[4];
    mma_bf16_zero(p, a.h, h0, h1);
    mma_bf16_16816(y.d[0], a.h, m0, m1);
    mma_bf16_16816(y.d[1], a.m, h0, h1);
    mma_bf16_16816(y.d[0], a.h, l0, l1);
    mma_bf16_16816(y.d[1], a.l, h0, h1);
    mma_bf16_16816(y.d[0], a.m, m0, m1);
#pragma unroll
    for (int e = 0; e < 4; ++e) y.s[e] += p[e];
}
__device__ __forceinline__ float ssd_total(const SsdSum& y, int e) { return y.s[e] + (y.d[0][e] + y.d[1][e]); }
// the three terms of a fragment lie 32 lanes x 16 bytes apart
__device__ __forceinline__ void ssd_load(SsdTerms& t, const uint4* at) {
    const uint4 h = at[0], m = at[32], l = at[64];
    t.h[0] = h.x; t.h[1] = h.y; t.h[2] = h.z; t.h[3] = h.w;
    t.m[0] = m.x; t.m[1] = m.y; t.m[2] = m.z; t.m[3] = m.w;
    t.l[0] = l.x; t.l[1] = l.y; t.l[2] = l.z; t.l[3] = l.w;
}

template <int NK>
__global__ void __launch_bounds__(kSsdWalk, 1) seq_ssd_walk_kernel(SsdBlockArgs p, int vec) {
    using Group = SsdGroup<NK>;
    constexpr int kX = kSsdBlock * kSsdLdx * 4, kHead = 3 * kSsdBlock * 4, kStage = Group::kBytes + kX + kHead, kSteps = NK / 16, kEighth = NK / 8, kTiles = kEighth / 8;
    extern __shared__ __align__(16) uint8_t sw_sm[];
    uint4* s_frag = reinterpret_cast<uint4*>(sw_sm + 2 * kStage);                      // S^T: [column tile][k-step][term][lane]
    uint4* x_frag = s_frag + 2 * kSteps * 96;                                         // x^T: [plain, scaled][column tile][k-step][term][lane]
    const sllm_seq_batch& b = p.b;
    const int seg = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * kSsdCols, grp = h / (p.heads / p.groups);
    const int start = b.seg_start[seg], len = b.seg_len[seg], slot = b.seg_slot[seg], blocks = (len + kSsdBlock - 1) / kSsdBlock;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3, ct = warp & 1, qu = warp >> 1;
    const size_t id0 = ssd_block_id(b.seg_tile0[seg], seg, 0);
    if (id0 + blocks > p.slots) {       // the scratch was sized by a tile count that leaves tokens out
        if (threadIdx.x == 0) *reinterpret_cast<volatile int32_t*>(p.status) = kStatusBatch;
        return;
    }
    const float* xs = p.x + (size_t)start * p.ldx + (size_t)h * p.dv + col0;
    auto issue = [&](int blk) {
        uint8_t* dst = sw_sm + (blk & 1) * kStage;
        const uint8_t* src = p.group_ws + ((id0 + blk) * p.groups + grp) * Group::kBytes;
        for (int i = threadIdx.x; i < Group::kBytes / 16; i += kSsdWalk) cp_async16(dst + 16 * i, src + 16 * i, 16);
        const int n = min(kSsdBlock, len - blk * kSsdBlock);
        float* dx = reinterpret_cast<float*>(dst + Group::kBytes);
        const float* xb = xs + (size_t)blk * kSsdBlock * p.ldx;
        if (vec) {
            for (int i = threadIdx.x; i < kSsdBlock * kSsdCols / 4; i += kSsdWalk) {
                const int tok = i / (kSsdCols / 4), j = (i % (kSsdCols / 4)) * 4;
                const bool has = tok < n && col0 + j < p.dv;
                cp_async16(dx + tok * kSsdLdx + j, has ? xb + (size_t)tok * p.ldx + j : p.x, has ? 16 : 0);
            }
        } else {
            for (int i = threadIdx.x; i < kSsdBlock * kSsdCols; i += kSsdWalk) {
                const int tok = i / kSsdCols, j = i % kSsdCols;
                const bool has = tok < n && col0 + j < p.dv;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dx + tok * kSsdLdx + j)), "l"(has ? xb + (size_t)tok * p.ldx + j : p.x), "r"(has ? 4 : 0)
                             : "memory");
            }
        }
        const float* hs = p.head_ws + ((id0 + blk) * p.heads + h) * (3 * kSsdBlock);
        if (threadIdx.x < kHead / 16) cp_async16(dst + Group::kBytes + kX + 16 * threadIdx.x, hs + 4 * threadIdx.x, 16);
        cp_async_commit();
    };
    if (blocks > 0) issue(0);
    // this warp's part of S^T: columns r0 / r1, states qu * kEighth + nt * 8 + 2c, + 1
    const int cl = ct * 16 + g, r0 = col0 + cl, r1 = r0 + 8;
    const bool ok0 = r0 < p.dv, ok1 = r1 < p.dv;
    float* st = p.state + ((size_t)slot * p.heads + h) * p.n_state * p.dv;
    float S[kTiles][4];
#pragma unroll
    for (int nt = 0; nt < kTiles; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = qu * kEighth + nt * 8 + 2 * c + (e & 1);
            S[nt][e] = (e < 2 ? ok0 : ok1) && row < p.n_state ? st[(size_t)row * p.dv + (e < 2 ? r0 : r1)] : 0.0f;
        }
    const float skip = p.skip ? p.skip[h] : 0.0f;
    for (int blk = 0; blk < blocks; ++blk) {
        cp_async_wait<0>();
        __syncthreads();                                     // the block has landed for everyone, and everyone has left the one before
        if (blk + 1 < blocks) issue(blk + 1);
        const uint8_t* rec = sw_sm + (blk & 1) * kStage;
        const float4* Cf = reinterpret_cast<const float4*>(rec) + lane;
        const float4* Bf = reinterpret_cast<const float4*>(rec + Group::kC) + lane;
        const float4* Wf = reinterpret_cast<const float4*>(rec + Group::kC + Group::kB) + lane;
        const float* sx = reinterpret_cast<const float*>(rec + Group::kBytes);
        const float* sG = reinterpret_cast<const float*>(rec + Group::kBytes + kX);
        const float* sL = sG + kSsdBlock;                    // second terms of the sums
        const float* sd = sL + kSsdBlock;
        const float Gn = sG[kSsdBlock - 1], Ln = sL[kSsdBlock - 1];
#pragma unroll
        for (int nt = 0; nt < kTiles; ++nt) {                // the state as halves of A fragments for all warps
            uint2 t[3];
            split3_bf16(S[nt][0], S[nt][1], t[0].x, t[1].x, t[2].x);
            split3_bf16(S[nt][2], S[nt][3], t[0].y, t[1].y, t[2].y);
            const int tile = qu * kTiles + nt;
            uint2* at = reinterpret_cast<uint2*>(s_frag + (ct * kSteps + tile / 2) * 96 + lane) + tile % 2;
#pragma unroll
            for (int i = 0; i < 3; ++i) at[64 * i] = t[i];
        }
        bool wild = false;                                   // a value is infinite or no number
        {                                                    // x^T as A fragments: a plain one or one decayed to the block's end per thread
            const int ks = qu & 3, scaled = qu >> 2;
            const float* at = sx + (ks * 16 + 2 * c) * kSsdLdx + cl;
            float v[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {                    // token 2c + (i & 1) + 8 (i >> 1): columns g and g + 8
                const int tok = ks * 16 + 2 * c + (i & 1) + 8 * (i >> 1);
                const float f = scaled ? exp2f((Gn - sG[tok]) + (Ln - sL[tok])) * sd[tok] : 1.0f;
                v[2 * i] = at[((i & 1) + 8 * (i >> 1)) * kSsdLdx] * f;
                v[2 * i + 1] = at[((i & 1) + 8 * (i >> 1)) * kSsdLdx + 8] * f;
            }
            // such a value would reach tokens before its own through the weights of zero that hide it from them: it is added by itself below
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (!ssd_finite(v[i])) {
                    wild = true;
                    v[i] = 0.0f;
                }
            uint4* to = x_frag + (scaled * 8 + ct * 4 + ks) * 96 + lane;
            uint4 t[3];
            split3_bf16(v[0], v[2], t[0].x, t[1].x, t[2].x);
            split3_bf16(v[1], v[3], t[0].y, t[1].y, t[2].y);
            split3_bf16(v[4], v[6], t[0].z, t[1].z, t[2].z);
            split3_bf16(v[5], v[7], t[0].w, t[1].w, t[2].w);
#pragma unroll
            for (int i = 0; i < 3; ++i) to[32 * i] = t[i];
        }
        wild = __syncthreads_or(wild);
        // outputs: columns of tile ct, tokens qu * 8 + 2c, + 1
        SsdSum y = {};
#pragma unroll
        for (int ks = 0; ks < kSteps; ++ks) {
            SsdTerms a;
            ssd_load(a, s_frag + (ct * kSteps + ks) * 96 + lane);
            ssd_mma(y, a, Cf[(qu * kSteps + ks) * 32]);
        }
        {
            const float2 G2 = *reinterpret_cast<const float2*>(sG + qu * 8 + 2 * c), L2 = *reinterpret_cast<const float2*>(sL + qu * 8 + 2 * c);
            const float e[2] = {exp2f(G2.x + L2.x), exp2f(G2.y + L2.y)};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                y.s[q] *= e[q & 1];
                y.d[0][q] *= e[q & 1];
                y.d[1][q] *= e[q & 1];
            }
        }
        const int i = qu * 8 + g;
        const float Gi = sG[i], Li = sL[i];
        for (int ks = 0; ks <= qu / 2; ++ks) {               // tokens j up to these
            SsdTerms a;
            ssd_load(a, x_frag + (ct * 4 + ks) * 96 + lane);
            const int j = ks * 16 + 2 * c;
            const float2 Ga = *reinterpret_cast<const float2*>(sG + j), Gb = *reinterpret_cast<const float2*>(sG + j + 8);
            const float2 La = *reinterpret_cast<const float2*>(sL + j), Lb = *reinterpret_cast<const float2*>(sL + j + 8);
            const float2 da = *reinterpret_cast<const float2*>(sd + j), db = *reinterpret_cast<const float2*>(sd + j + 8);
            const float4 w = Wf[ssd_w_tile(qu, ks) * 32];
            const float w0 = j <= i ? w.x * (exp2f((Gi - Ga.x) + (Li - La.x)) * da.x) : 0.0f, w1 = j + 1 <= i ? w.y * (exp2f((Gi - Ga.y) + (Li - La.y)) * da.y) : 0.0f;
            const float w2 = j + 8 <= i ? w.z * (exp2f((Gi - Gb.x) + (Li - Lb.x)) * db.x) : 0.0f, w3 = j + 9 <= i ? w.w * (exp2f((Gi - Gb.y) + (Li - Lb.y)) * db.y) : 0.0f;
            ssd_mma(y, a, make_float4(w0, w1, w2, w3));
        }
        if (wild) {
            const float* W = reinterpret_cast<const float*>(rec + Group::kC + Group::kB);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tok = qu * 8 + 2 * c + (e & 1);
                for (int j = 0; j <= tok; ++j) {
                    const float v = sx[j * kSsdLdx + cl + (e < 2 ? 0 : 8)];
                    if (ssd_finite(v)) continue;
                    const float w = W[(ssd_w_tile(qu, j / 16) * 32 + (tok & 7) * 4 + j % 8 / 2) * 4 + j % 16 / 8 * 2 + j % 2];
                    y.s[e] = fmaf(w * (exp2f((sG[tok] - sG[j]) + (sL[tok] - sL[j])) * sd[j]), v, y.s[e]);
                }
            }
        }
        const int n = min(kSsdBlock, len - blk * kSsdBlock);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int tok = qu * 8 + 2 * c + (e & 1);
            if (tok < n && (e < 2 ? ok0 : ok1))
                p.y[(size_t)(start + blk * kSsdBlock + tok) * p.ldy + (size_t)h * p.dv + (e < 2 ? r0 : r1)] = fmaf(skip, sx[tok * kSsdLdx + cl + (e < 2 ? 0 : 8)], ssd_total(y, e));
        }
        // the state
        const float dn = exp2f(Gn + Ln);
        SsdSum add[kTiles] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            SsdTerms a;
            ssd_load(a, x_frag + (2 * 4 + ct * 4 + ks) * 96 + lane);
#pragma unroll
            for (int nt = 0; nt < kTiles; ++nt) ssd_mma(add[nt], a, Bf[((qu * kTiles + nt) * 4 + ks) * 32]);
        }
        if (wild) {
            const float* B = reinterpret_cast<const float*>(rec + Group::kC);
#pragma unroll
            for (int nt = 0; nt < kTiles; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    for (int j = 0; j < n; ++j) {
                        const float f = exp2f((Gn - sG[j]) + (Ln - sL[j])) * sd[j], v = sx[j * kSsdLdx + cl + (e < 2 ? 0 : 8)] * f;
                        if (!ssd_finite(v)) add[nt].s[e] = fmaf(B[(((qu * kTiles + nt) * 4 + j / 16) * 32 + (2 * c + (e & 1)) * 4 + j % 8 / 2) * 4 + j % 16 / 8 * 2 + j % 2], v, add[nt].s[e]);
                    }
        }
#pragma unroll
        for (int nt = 0; nt < kTiles; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[nt][e] = fmaf(dn, S[nt][e], ssd_total(add[nt], e));
    }
#pragma unroll
    for (int nt = 0; nt < kTiles; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = qu * kEighth + nt * 8 + 2 * c + (e & 1);
            if ((e < 2 ? ok0 : ok1) && row < p.n_state) st[(size_t)row * p.dv + (e < 2 ? r0 : r1)] = S[nt][e];
        }
}

template <int NK>
static int launch_ssd(SsdBlockArgs p, cudaStream_t st) {
    using Group = SsdGroup<NK>;
    auto aligned = [](const void* q) { return ((uintptr_t)q % 16) == 0; };
    const int vec_prep = p.n_state % 4 == 0 && p.ldb % 4 == 0 && p.ldc % 4 == 0 && aligned(p.B) && aligned(p.C);
    const int vec = p.dv % 4 == 0 && p.ldx % 4 == 0 && aligned(p.x);
    constexpr int smem_prep = (2 * kSsdBlock * (NK + 4) + kSsdBlock * (kSsdBlock + 1)) * 4;
    constexpr int smem = 2 * (Group::kBytes + kSsdBlock * kSsdLdx * 4 + 3 * kSsdBlock * 4) + 2 * (NK / 16) * 96 * 16 + 2 * 2 * 4 * 96 * 16;
    static bool sized = false;
    if (!sized) {
        SLLM_CUDA(cudaFuncSetAttribute(seq_ssd_prepare_kernel<NK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_prep));
        SLLM_CUDA(cudaFuncSetAttribute(seq_ssd_walk_kernel<NK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        sized = true;
    }
    const int per = kSsdThreads / 32;
    seq_ssd_prepare_kernel<NK><<<dim3((unsigned)p.slots, p.groups + (p.heads + per - 1) / per), kSsdThreads, smem_prep, st>>>(p, vec_prep);
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    seq_ssd_walk_kernel<NK><<<dim3(p.b.nseg, p.heads, (p.dv + kSsdCols - 1) / kSsdCols), kSsdWalk, smem, st>>>(p, vec);
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}

}  // namespace sllm

using namespace sllm;

extern "C" int64_t sllm_seq_ssd_block_ws_bytes(int32_t n_qtiles, int32_t nseg, int32_t heads, int32_t groups, int32_t n_state) {
    if (n_qtiles <= 0 || nseg <= 0 || heads <= 0 || groups <= 0 || n_state <= 0 || n_state > kSsdMaxState) return 0;
    return (int64_t)ssd_block_count(n_qtiles, nseg) * ((int64_t)groups * ssd_block_group_bytes(n_state <= 64 ? 64 : 128) + (int64_t)heads * 3 * kSsdBlock * 4);
}

extern "C" int sllm_seq_ssd_blocks(const sllm_seq_batch* b, const float* x, int32_t ldx, const float* B, int32_t ldb, const float* C, int32_t ldc, const float* step_logit,
                                   int32_t lda, const float* A_log, const float* dt_bias, const float* skip, int32_t heads, int32_t groups, int32_t n_state, int32_t dv,
                                   float* state, float* y, int32_t ldy, const float* conv_x, int32_t ld_conv, int32_t channels, int32_t taps, float* ring, void* block_ws,
                                   sllm_stream_t stream) {
    SLLM_REQUIRE(b && b->T > 0 && b->nseg > 0 && b->seg_start && b->seg_len && b->seg_slot && b->seg_tile0 && (long long)b->n_qtiles * 32 >= b->T, SLLM_EINVAL,
                 "seq_ssd_blocks: incomplete batch description");
    SLLM_REQUIRE(x && B && C && step_logit && A_log && dt_bias && state && y && block_ws && ((uintptr_t)block_ws % 16) == 0, SLLM_EINVAL, "seq_ssd_blocks: bad argument");
    SLLM_REQUIRE(heads > 0 && groups > 0 && heads % groups == 0 && n_state > 0 && dv > 0, SLLM_EINVAL, "seq_ssd_blocks: %d heads over %d groups", heads, groups);
    SLLM_REQUIRE(n_state <= kSsdMaxState && heads <= 65535 && groups + heads / 8 < 65535, SLLM_ENOTSUP, "seq_ssd_blocks: %d states per channel beyond %d", n_state, kSsdMaxState);
    SLLM_REQUIRE(!ring || taps <= 1 || conv_x, SLLM_EINVAL, "seq_ssd_blocks: a ring without its inputs");
    SsdBlockArgs p{*b, x, B, C, step_logit, ldx, ldb, ldc, lda, A_log, dt_bias, skip, heads, groups, n_state, dv, state, y, ldy, nullptr, ssd_block_count(b->n_qtiles, b->nseg), nullptr, nullptr};
    if (int rc = status_word(&p.status)) return rc;
    p.group_ws = reinterpret_cast<uint8_t*>(block_ws);
    p.head_ws = reinterpret_cast<float*>(p.group_ws + p.slots * groups * ssd_block_group_bytes(n_state <= 64 ? 64 : 128));
    if (int rc = n_state <= 64 ? launch_ssd<64>(p, as_stream(stream)) : launch_ssd<128>(p, as_stream(stream))) return rc;
    return ring && taps > 1 ? sllm_seq_ring_store(b, conv_x, ld_conv, channels, taps, ring, stream) : SLLM_OK;
}
