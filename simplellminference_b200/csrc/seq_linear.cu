// csrc/seq_linear.cu — sllm_seq_linear: C = alpha * (A . W^T + bias) (+ C) for the ragged token batch. Three bodies:
//   * rows kernels (T <= 8, decode-sized steps): every weight streamed once past activations in registers, bf16 ones of several rows through the tensor cores; a body without that
//     set-up for small matrices, with scalar loads where 16-byte accesses do not fit;
//   * tile_kernel  (any shape): 64 x 64 x 16 shared-memory tiles, 4 x 4 outputs per thread, fp32 FMAs with fp32 accumulation. This is
//     the body of the all-fp32 mode, and of bf16 products whose shape the tensor-core tiles do not take;
//   * the tcgen05 GEMM of the prefill path (prefill_gemm.cu) for bf16 weights when the caller passes a bf16 scratch for A and the shape
//     fits its TMA boxes; without a scale the GEMM's own epilogue adds the bias and stores (or adds) into C, otherwise bias, alpha and accumulation
//     run as a short epilogue kernel over C.
// In bf16 mode (round_a) the activations are rounded to bf16 as they are loaded, so all three bodies multiply the same operands and
// differ only in summation order.
#include <climits>
#include <type_traits>

#include "prefill.cuh"
#include "seq_attn.cuh"

namespace sllm {

struct LinArgs {
    const float* A; const void* W; const float* bias; float* C;
    int lda, ldw, ldc, T, N, K, w_dtype, accumulate, round_a;
    float alpha;
    long long a_bs, w_bs, bias_bs, c_bs;
    const int32_t* rows_dev;   // device memory or NULL: rows from rows_dev[b * rows_bs] on are not computed (tile body and tensor cores)
    const int32_t* w_index;    // rows body, device memory or NULL: product b of the batch uses matrix w_index[b] (W + w_index[b] * w_bs); -1 = no matrix, zeros
    int a_div;                 // rows body: product b reads the activations of batch element b / a_div (0 or 1: its own)
    int rows_bs;               // tile body: 1 = a row count per product of the batch
    int w_fixed;               // rows bodies: no kernel of the same captured graph writes W, whose first rows are asked for before the wait for the kernel in front (and for all before it)
};

constexpr int kRowsMax = 8;
constexpr int kRowsBlock = 64;     // weight rows between two flushes of the partial sums

// TT: activation rows the products are computed for (T rounded up to 1, 2, 4 or 8). A lane owns two 16-byte chunks of every weight row of a panel
// of K and keeps the matching activations of all TT rows in registers (8 rows: half as many warps, so that they fit); kGroup weight rows are
// reduced across the lanes together; kDeep rows are in flight per warp: a ring of 64 KB per SM (8 rows: 128 KB), where the HBM rate asks for some 35 at
// its latency. Groups of two, not four: less code to fetch at the start of every launch (2048 x 2048, one row 5.2 -> 4.7 us; 6144 x 4096, four
// rows 16.5 -> 14.6 us).
template <int TT>
struct RowsShape {
    static constexpr int kWarps = TT <= 4 ? 16 : 8, kChunks = 2, kGroup = 2, kDeep = TT <= 4 ? 4 : 16;
    static constexpr int kRing = kWarps * kDeep * kChunks * 512;
};

// Up to 8 activation rows against a stream of weight rows. Bound: HBM, every weight is read once. One CTA per SM takes a contiguous
// share of the weight rows; WK = 2^wk_log2 of its warps cut K among themselves (so that every SM's share ends at the same time whatever N), the
// others take other rows. What a weight costs beside its load was the bound of a body whose lanes read the activations from memory for every weight
// row (2 T bytes of activations through L1 per byte of weights: 1.1 TB/s at 4 rows of 6144 x 4096 bf16, now 3.4; one row 2.6, now 4.4 and 5.3 at
// 32000 x 2048): here the activations of a lane's columns stay in registers for all rows, the
// weights arrive through cp.async in a ring that only their own lane reads back (no barrier in the stream), fma.rn.f32x2 does two products per
// instruction, and TT x kGroup sums cross the lanes in one halving exchange.
template <int WD, int TT>
__global__ void __launch_bounds__(RowsShape<TT>::kWarps * 32, 1) seq_linear_rows_kernel(LinArgs p, int wk_log2) {
    using Shape = RowsShape<TT>;
    constexpr int E = WD == SLLM_BF16 ? 8 : 4;                 // weights per 16-byte chunk
    constexpr int C = Shape::kChunks, RG = Shape::kGroup, D = Shape::kDeep, V = RG * TT;
    extern __shared__ __align__(16) uint8_t rows_smem[];
    const int b = blockIdx.y;
    const bool early = p.w_fixed && !p.w_index;
    if (!early) after_previous();
    const int wb = p.w_index ? p.w_index[b] : b;               // which matrix of W; negative: none (the outputs are zeros)
    const float* A = p.A + (size_t)(p.a_div > 1 ? b / p.a_div : b) * p.a_bs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int WK = 1 << wk_log2, WR = Shape::kWarps >> wk_log2, wk = warp & (WK - 1), wr = warp >> wk_log2;
    const int n_lo = (int)((long long)p.N * blockIdx.x / gridDim.x), rows = (int)((long long)p.N * (blockIdx.x + 1) / gridDim.x) - n_lo;
    const int chunks = wb >= 0 ? p.K / E : 0, panel = WK * 32 * C, panels = max(1, (chunks + panel - 1) / panel);
    const int blocks = (rows + kRowsBlock - 1) / kRowsBlock;
    const size_t row_bytes = (size_t)p.ldw * (16 / E);
    const uint8_t* w = reinterpret_cast<const uint8_t*>(p.W) + ((size_t)max(wb, 0) * p.w_bs) * (16 / E) + (size_t)(n_lo + wr) * row_bytes;
    const uint32_t ring = smem_u32(rows_smem) + warp * (D * C * 512) + lane * 16;
    float* table = reinterpret_cast<float*>(rows_smem + Shape::kRing);      // [2][WK][kRowsBlock][TT]

    // Weight rows in the order in which they are consumed: per block of rows, per panel of K, the warp's rows in groups of RG. `run` counts the rows
    // of the current (block, panel) that are still to be asked for; rows that only fill up a group are not fetched and their sums not used.
    int i_blk = 0, i_pan = 0, run = 0, pad = 0;
    const uint8_t* src = w;
    uint32_t off[C], bytes[C], fill = ring;
    const size_t step = row_bytes << (__ffs(WR) - 1);
    auto begin_run = [&]() {
        const int cur = min(kRowsBlock, rows - i_blk * kRowsBlock);
        run = max(0, (cur - wr + WR - 1) / WR);
        pad = ((cur + WR - 1) / WR + RG - 1) / RG * RG - run;
        src = w + (size_t)i_blk * kRowsBlock * row_bytes;
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const int ch = i_pan * panel + (j * WK + wk) * 32 + lane;
            off[j] = ch < chunks ? ch * 16 : 0;
            bytes[j] = ch < chunks ? 16 : 0;
        }
    };
    auto issue = [&]() {
        if (run > 0) {
#pragma unroll
            for (int j = 0; j < C; ++j)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(fill + j * 512), "l"(src + off[j]), "r"(bytes[j]) : "memory");
            src += step;
            --run;
        } else {
            --pad;
        }
        fill = fill + C * 512 == ring + D * C * 512 ? ring : fill + C * 512;
        cp_async_commit();
        if (run + pad == 0 && i_blk < blocks) {
            if (++i_pan == panels) {
                i_pan = 0;
                ++i_blk;
            }
            if (i_blk < blocks) begin_run();
            else pad = 1 << 30;          // nothing left: empty groups from here on
        }
    };
    // the activations of this lane's columns of a panel
    uint64_t act[TT][C][E / 2];
    auto load_act = [&](int pan) {
#pragma unroll
        for (int t = 0; t < TT; ++t)
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const int ch = pan * panel + (j * WK + wk) * 32 + lane;
                const bool ok = t < p.T && ch < chunks;
#pragma unroll
                for (int e = 0; e < E; e += 4) {
                    float4 a = ok ? *reinterpret_cast<const float4*>(A + (size_t)t * p.lda + (size_t)ch * E + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p.round_a) a = make_float4(seq_round_bf16(a.x), seq_round_bf16(a.y), seq_round_bf16(a.z), seq_round_bf16(a.w));
                    act[t][j][e / 2] = pair_f32(a.x, a.y);
                    act[t][j][e / 2 + 1] = pair_f32(a.z, a.w);
                }
            }
    };
    if (blocks) begin_run(); else pad = 1 << 30;
    // Half of the ring is asked for before the activations, the rest behind them; eight rows, whose activations take longer, ask for all of it. Measured against asking for all of it,
    // launches one behind the other, means over nine shapes: one to four bf16 rows 2 to 3 % shorter, fp32 1 to 2 %; captured steps of one to four requests 0.3 to 3 % shorter, of
    // eight (half, then the rest) 0 to 2 % longer.
    constexpr int kFirst = TT == 8 ? D : D / 2;
#pragma unroll
    for (int i = 0; i < kFirst; ++i) issue();
    if (early) after_previous();
    load_act(0);
#pragma unroll
    for (int i = kFirst; i < D; ++i) issue();

    // after the exchange a lane holds the sum of row `which / TT` of the group and activation row `which % TT`
    int which = 0;
#pragma unroll
    for (int n = V / 2, bit = 16; n >= 1; n /= 2, bit /= 2) which = which * 2 + ((lane & bit) ? 1 : 0);
    const bool writes = lane % (32 / V) == 0;
    uint32_t slot = ring;
    for (int blk = 0; blk < blocks; ++blk) {
        const int cur = min(kRowsBlock, rows - blk * kRowsBlock), steps = (cur + WR - 1) / WR;
        float* tab = table + (size_t)(blk & 1) * (WK * kRowsBlock * TT);
        for (int pan = 0; pan < panels; ++pan) {
            if (pan + blk > 0 && panels > 1) load_act(pan);
            float* cell = tab + (size_t)(wk * kRowsBlock + (which / TT) * WR + wr) * TT + which % TT;
            for (int g = 0; g < steps; g += RG, cell += RG * WR * TT) {
                cp_async_wait<D - RG>();
                uint64_t acc[RG][TT];
                uint4 us[2][C];       // two rows' chunks on their way (D is a multiple of RG: a group's slots are adjacent)
                auto fetch = [&](int r) {
#pragma unroll
                    for (int j = 0; j < C; ++j)
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(us[r & 1][j].x), "=r"(us[r & 1][j].y), "=r"(us[r & 1][j].z), "=r"(us[r & 1][j].w)
                                     : "r"(slot + (r * C + j) * 512)
                                     : "memory");
                };
                fetch(0);
#pragma unroll
                for (int r = 0; r < RG; ++r) {
                    if (r + 1 < RG) fetch(r + 1);
#pragma unroll
                    for (int t = 0; t < TT; ++t) acc[r][t] = 0ull;
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        const uint4 u = us[r & 1][j];
                        uint64_t wv[E / 2];
                        if (WD == SLLM_BF16) {
                            wv[0] = pair_f32(u.x << 16, u.x & 0xffff0000u);
                            wv[1] = pair_f32(u.y << 16, u.y & 0xffff0000u);
                            wv[E / 2 - 2] = pair_f32(u.z << 16, u.z & 0xffff0000u);
                            wv[E / 2 - 1] = pair_f32(u.w << 16, u.w & 0xffff0000u);
                        } else {
                            wv[0] = pair_f32(u.x, u.y);
                            wv[1] = pair_f32(u.z, u.w);
                        }
#pragma unroll
                        for (int t = 0; t < TT; ++t)
#pragma unroll
                            for (int e = 0; e < E / 2; ++e) fma_pair(acc[r][t], wv[e], act[t][j][e]);
                    }
                }
                slot = slot + RG * C * 512 == ring + D * C * 512 ? ring : slot + RG * C * 512;
#pragma unroll
                for (int r = 0; r < RG; ++r) issue();
                // V sums over 32 lanes: in every step a lane keeps half of its values and gets the partner's part of them
                float v[V];
#pragma unroll
                for (int r = 0; r < RG; ++r)
#pragma unroll
                    for (int t = 0; t < TT; ++t) v[r * TT + t] = pair_sum(acc[r][t]);
#pragma unroll
                for (int n = V / 2, bit = 16; n >= 1; n /= 2, bit /= 2) {
                    const bool up = lane & bit;
#pragma unroll
                    for (int i = 0; i < n; ++i) {
                        const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                    }
                }
#pragma unroll
                for (int o = 16 / V; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
                if (writes && (g + which / TT) * WR + wr < kRowsBlock) *cell = pan ? *cell + v[0] : v[0];
            }
        }
        __syncthreads();
        const float* bias = p.bias ? p.bias + (size_t)b * p.bias_bs : nullptr;
        float* out = p.C + (size_t)b * p.c_bs;
        for (int o = threadIdx.x; o < cur * p.T; o += Shape::kWarps * 32) {
            const int t = o / cur, r = o % cur, n = n_lo + blk * kRowsBlock + r;
            float sum = 0.0f;
            for (int k = 0; k < WK; ++k) sum += tab[(size_t)(k * kRowsBlock + r) * TT + t];
            const float val = p.alpha * (sum + (bias ? bias[n] : 0.0f));
            float* c = out + (size_t)t * p.ldc + n;
            *c = p.accumulate ? *c + val : val;
        }
    }
}

// Up to 8 activation rows, rounded to bf16, against a stream of bf16 weight rows on the tensor cores: mma.sync m16n8k16 with 8 weight rows as the columns. Bound: HBM, every weight is read
// once. One CTA per SM takes a contiguous share of the weight rows; WK = 2^wk_log2 of its 16 warps cut K among themselves, 256 columns each of a panel of K, the others take other
// tiles of 8 rows. The activations stay in registers; the weights arrive through cp.async in a ring of each warp's own, 16 rows of 512 bytes (128 KB an SM), and leave it through ldmatrix.
// A weight costs a fortieth of an instruction of each kind where fma.rn.f32x2 and the exchange between lanes took a tenth, and the same for one row as for eight.
// Accuracy: the tensor core truncates its sums. So an activation is split into its upper and its lower four significant bits, which go through as rows 0..7 and 8..15: products of 12
// bits, whose sums of 16 fit a result's 24 but for columns 2^8 below the largest; each starts from zero and is added with ordinary rounding, and the warps' sums meet in double.
// Error against float64, streaming body | this one: 8.2e-8 | 5.4e-8 (K = 4096), 1.03e-7 | 6.4e-8 (11008), 5.5e-8 | 5.1e-8 (264); unsplit it was 9.9e-8.
constexpr int kMmaWarps = 16, kMmaSlice = 256, kMmaSteps = kMmaSlice / 32, kMmaHalves = 4, kMmaHalf = 4 * 2 * kMmaSlice, kMmaRing = kMmaHalves * kMmaHalf, kMmaStage = 8 * kMmaSlice;      // bytes: half a tile, ring of a warp, half of its columns' activations
__host__ __device__ __forceinline__ int mma_block_rows(int WR) { return WR <= 2 ? 48 : WR <= 8 ? 64 : 128; }      // weight rows between two flushes of the partial sums: whole rounds of tiles
// a pair of bf16 values as a pair of their upper four significant bits and one of the lower four
__device__ __forceinline__ void mma_halves(uint32_t a, uint32_t& hi, uint32_t& lo) {
    hi = a & 0xfff0fff0u;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(hi));
}
__device__ __forceinline__ void mma_fragments(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// A warp's results whose sums (in `tab`) are no number, once more: in fp32 from operands that are not split, a result at a time by all lanes.
static __device__ __noinline__ void mma_unsplit(const LinArgs& p, const float* a, const uint16_t* W, const float* bias, float* out, const float* tab, int ldt, int WK, int n, int n0, int K) {
    const int lane = threadIdx.x & 31;
    for (int r0 = 4 * ((threadIdx.x >> 5) & 8); r0 < n; r0 += 64) {
        double sum = 0.0;
        for (int k = 0; r0 + lane < n && k < WK; ++k) sum += (double)tab[(size_t)k * 8 * ldt + r0 + lane];
        for (uint32_t none = __ballot_sync(0xffffffffu, sum != sum); none; none &= none - 1) {
            const int at = n0 + r0 + __ffs(none) - 1;
            const uint16_t* w = W + (size_t)at * p.ldw;
            float acc = 0.0f;
            for (int k = 4 * lane; k < K; k += 128) {
                const float4 x = *reinterpret_cast<const float4*>(a + k);
                const uint2 u = *reinterpret_cast<const uint2*>(w + k);
                acc = fmaf(seq_round_bf16(x.x), bf16_lo(u.x), fmaf(seq_round_bf16(x.y), bf16_hi(u.x), fmaf(seq_round_bf16(x.z), bf16_lo(u.y), fmaf(seq_round_bf16(x.w), bf16_hi(u.y), acc))));
            }
            acc = warp_sum(acc);
            if (lane == 0) {
                const float val = p.alpha * (acc + (bias ? bias[at] : 0.0f));
                out[at] = p.accumulate ? out[at] + val : val;
            }
        }
    }
}
__global__ void __launch_bounds__(kMmaWarps * 32, 1) seq_linear_rows_mma_kernel(const __grid_constant__ LinArgs p, int wk_log2) {
    extern __shared__ __align__(16) uint8_t mma_smem[];        // rings, 2 KB a warp for activations on their way, then [2][WK][8 activation rows][block + 8] partial sums
    const int b = blockIdx.y;
    const bool early = p.w_fixed && !p.w_index;
    if (!early) after_previous();
    const int wb = p.w_index ? p.w_index[b] : b;               // which matrix of W; negative: none (the outputs are zeros)
    const float* A = p.A + (size_t)(p.a_div > 1 ? b / p.a_div : b) * p.a_bs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int WK = 1 << wk_log2, WR = kMmaWarps >> wk_log2, wk = warp & (WK - 1), wr = warp >> wk_log2, block = mma_block_rows(WR), ldt = block + 8;
    const int n_lo = (int)((long long)p.N * blockIdx.x / gridDim.x), rows = (int)((long long)p.N * (blockIdx.x + 1) / gridDim.x) - n_lo;
    const int K = wb >= 0 ? p.K : 0, panel = WK * kMmaSlice, panels = max(1, (K + panel - 1) / panel), blocks = (rows + block - 1) / block;
    const uint32_t ring = smem_u32(mma_smem) + warp * kMmaRing;
    float* table = reinterpret_cast<float*>(mma_smem + kMmaWarps * (kMmaRing + kMmaStage));

    struct Unit { int blk, pan, row; };                        // a tile of this warp: block, panel, first row in the block
    auto settle = [&](Unit& x) {                               // on to one that has rows, or past the last block
        while (x.blk < blocks && x.row >= min(block, rows - x.blk * block)) {
            x.row = 8 * wr;
            if (++x.pan == panels) {
                x.pan = 0;
                ++x.blk;
            }
        }
    };
    Unit u{0, 0, 8 * wr};
    settle(u);
    Unit ahead = u;                                            // the tile being asked for, half by half
    int half = 0;
    uint32_t fill = ring;
    // this lane's 16 bytes of weight row 0
    const uint8_t* W = reinterpret_cast<const uint8_t*>(p.W) + (((size_t)max(wb, 0) * p.w_bs + (size_t)n_lo * p.ldw + wk * kMmaSlice + 8 * lane) << 1);
    const size_t row_bytes = (size_t)p.ldw * 2;
    const int K0 = K - wk * kMmaSlice - 8 * lane;              // columns from there on
    auto issue = [&]() {
        if (ahead.blk < blocks) {
            const int row = ahead.blk * block + ahead.row + 4 * half;
            const int left = ahead.pan * panel < K0 ? rows - row : 0;      // rows that are there
            const uint8_t* src = left > 0 ? W + row * row_bytes + (size_t)(2 * ahead.pan * panel) : reinterpret_cast<const uint8_t*>(p.W);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(fill + r * (2 * kMmaSlice) + ((lane ^ (4 * half + r)) << 4)), "l"(src), "r"(r < left ? 16 : 0) : "memory");
                if (r + 1 < left) src += row_bytes;
            }
            if (half) {
                ahead.row += 8 * WR;
                settle(ahead);
            }
            half ^= 1;
            fill = fill + kMmaHalf == ring + kMmaRing ? ring : fill + kMmaHalf;
        }
        cp_async_commit();
    };
    const int mr = lane & 7;                                   // row of this lane's addresses for ldmatrix, and its 16-byte piece, swizzled
    const uint32_t piece = (uint32_t)(((lane >> 3) ^ mr) << 4);
    // The activations of this warp's columns as fragments: rows of 128 columns at a time through shared memory (a load of 8 bytes per lane and fragment touched eight lines each: 2 us
    // for eight rows of 4096). Rows from T on hold what is there: they meet no other row.
    uint32_t act[kMmaSteps][4];
    auto load_act = [&](int pan) {
        const uint32_t stage = smem_u32(mma_smem) + kMmaWarps * kMmaRing + warp * kMmaStage;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = pan * panel + wk * kMmaSlice + h * (kMmaSlice / 2) + 4 * lane;
            float4 x[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) x[t] = t < p.T && k < K ? *reinterpret_cast<const float4*>(A + (size_t)t * p.lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            __syncwarp();
#pragma unroll
            for (int t = 0; t < 8; ++t)
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(stage + t * kMmaSlice + (((lane >> 1) ^ t) << 4) + (lane & 1) * 8), "r"(pack_bf16(x[t].x, x[t].y)),
                             "r"(pack_bf16(x[t].z, x[t].w)) : "memory");
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kMmaSteps / 2; ++i) mma_fragments(act[h * (kMmaSteps / 2) + i], stage + mr * kMmaSlice + (piece ^ (64u * i)));
        }
    };
#pragma unroll
    for (int i = 0; i < kMmaHalves; ++i) issue();
    if (early) after_previous();
    load_act(0);
    uint32_t take = ring;
    for (int blk = 0; blk < blocks; ++blk) {
        const int n = min(block, rows - blk * block);
        float* tab = table + (size_t)(blk & 1) * WK * 8 * ldt;
        for (int pan = 0; pan < panels; ++pan) {
            if (panels > 1 && pan + blk > 0) load_act(pan);
            while (u.blk == blk && u.pan == pan) {
                cp_async_wait<kMmaHalves - 2>();
                __syncwarp();
                const uint32_t second = take + kMmaHalf == ring + kMmaRing ? ring : take + kMmaHalf;
                const uint32_t from = (mr < 4 ? take : second) + (mr & 3) * (2 * kMmaSlice);
                float s[4] = {};
#pragma unroll
                for (int i = 0; i < kMmaSteps; ++i) {
                    uint32_t w[4];                             // columns 32 i + 8 m + 2 c, + 1 of weight row g
                    mma_fragments(w, from + (piece ^ (64u * i)));
#pragma unroll
                    for (int m = 0; m < 4; m += 2) {
                        float d[4];
                        uint32_t a[4];
                        mma_halves(act[i][m], a[0], a[1]);
                        mma_halves(act[i][m + 1], a[2], a[3]);
                        mma_bf16_zero(d, a, w[m], w[m + 1]);
#pragma unroll
                        for (int q = 0; q < 4; ++q) s[q] += d[q];
                    }
                }
                __syncwarp();
                issue();
                issue();
                take = second + kMmaHalf == ring + kMmaRing ? ring : second + kMmaHalf;
                float2* cell = reinterpret_cast<float2*>(tab + (size_t)(wk * 8 + g) * ldt + u.row + 2 * c);
                float2 v = make_float2(s[0] + s[2], s[1] + s[3]);
                if (pan) {
                    const float2 o = *cell;
                    v = make_float2(o.x + v.x, o.y + v.y);
                }
                *cell = v;
                u.row += 8 * WR;
                settle(u);
            }
        }
        __syncthreads();
        const float* bias = p.bias ? p.bias + (size_t)b * p.bias_bs : nullptr;
        float* out = p.C + (size_t)b * p.c_bs;
        // a warp has one activation row and every other 32 columns
        const int t = warp & 7;
        bool missing = false;
        for (int r = 4 * (warp & 8) + lane; t < p.T && r < n; r += 64) {
            const int at = n_lo + blk * block + r;
            double sum = 0.0;
#pragma unroll 4
            for (int k = 0; k < WK; ++k) sum += (double)tab[(size_t)(k * 8 + t) * ldt + r];
            if (__builtin_expect(sum != sum, 0)) {
                missing = true;
                continue;
            }
            const float val = p.alpha * ((float)sum + (bias ? bias[at] : 0.0f));
            float* to = out + (size_t)t * p.ldc + at;
            *to = p.accumulate ? *to + val : val;
        }
        // An infinite activation has no lower half (inf - inf), and an infinite weight times a lower half of zero is no number either, where the product itself would be infinite
        if (__builtin_expect(__any_sync(0xffffffffu, missing), 0))
            mma_unsplit(p, A + (size_t)t * p.lda, reinterpret_cast<const uint16_t*>(p.W) + (size_t)max(wb, 0) * p.w_bs, bias, out + (size_t)t * p.ldc, tab + (size_t)t * ldt, ldt, WK, n,
                        n_lo + blk * block, K);
    }
}

constexpr int kInFlight = 2;   // 16-byte weight loads per batch and lane; two batches are in flight (measured: 2 x 2 at four resident CTAs beats 1 x 4 by 12 %)

// Small matrices (launch_rows says which) and accesses that are not 16 bytes wide: `wpr` warps (1, 2, 4 or 8) share one output column and cut K among them, so that a matrix with few rows and long rows still fills the
// machine; a lane keeps two batches of 16-byte weight loads in flight (the next batch travels while this one is multiplied). The partial sums of a column meet in shared memory in a fixed order.
// kShort: a load's products are summed before they join the sum of a lane, as many roundings in a row as in the streaming body (error of fp32 1000 x 11008 at five rows
// 1.13e-7, else 1.2e-7; streaming 1.08e-7), for the larger ones of these products; 2 to 8 % slower, so not for the others.
template <int WD, bool kShort>
__global__ void __launch_bounds__(256, 4) seq_linear_rows_small_kernel(LinArgs p, int vec, int wpr) {
    __shared__ float part_sum[8][kRowsMax];
    const int b = blockIdx.y;
    const bool early = p.w_fixed && !p.w_index && vec;
    if (!early) after_previous();
    const int wb = p.w_index ? p.w_index[b] : b;             // which matrix of W; negative: none (the outputs are zeros)
    const float* A = p.A + (size_t)(p.a_div > 1 ? b / p.a_div : b) * p.a_bs;
    const float* bias = p.bias ? p.bias + (size_t)b * p.bias_bs : nullptr;
    float* C = p.C + (size_t)b * p.c_bs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * 8 + warp, n = item / wpr, part = item % wpr;
    constexpr int E = WD == SLLM_BF16 ? 8 : 4;                 // weights per 16-byte load
    const int kper = ((p.K + wpr - 1) / wpr + E - 1) / E * E;  // this warp's share of K, a multiple of the load width
    const int k_lo = part * kper, k_hi = min(p.K, k_lo + kper);
    float acc[kRowsMax];
#pragma unroll
    for (int t = 0; t < kRowsMax; ++t) acc[t] = 0.0f;
    if (n < p.N && wb >= 0) {
        if (vec) {
            const uint8_t* w = reinterpret_cast<const uint8_t*>(p.W) + ((size_t)wb * p.w_bs + (size_t)n * p.ldw) * (16 / E);
            constexpr int kStep = kInFlight * 32 * E;
            auto load = [&](uint4 (&u)[kInFlight], int k0) {
#pragma unroll
                for (int j = 0; j < kInFlight; ++j) {
                    const int k = k0 + j * 32 * E;
                    u[j] = k < k_hi ? ld_stream(w + (size_t)k * (16 / E)) : make_uint4(0u, 0u, 0u, 0u);     // W may be the work of the kernel in front
                }
            };
            auto consume = [&](const uint4 (&u)[kInFlight], int k0) {
#pragma unroll
                for (int j = 0; j < kInFlight; ++j) {
                    const int k = k0 + j * 32 * E;
                    if (k < k_hi) {
                        float wv[E];
                        if (WD == SLLM_BF16) {
                            wv[0] = bf16_lo(u[j].x); wv[1] = bf16_hi(u[j].x); wv[2] = bf16_lo(u[j].y); wv[3] = bf16_hi(u[j].y);
                            wv[E - 4] = bf16_lo(u[j].z); wv[E - 3] = bf16_hi(u[j].z); wv[E - 2] = bf16_lo(u[j].w); wv[E - 1] = bf16_hi(u[j].w);
                        } else {
                            wv[0] = __uint_as_float(u[j].x); wv[1] = __uint_as_float(u[j].y); wv[2] = __uint_as_float(u[j].z); wv[3] = __uint_as_float(u[j].w);
                        }
#pragma unroll
                        for (int t = 0; t < kRowsMax; ++t) {
                            if (t < p.T) {
                                const float* ar = A + (size_t)t * p.lda + k;
                                float sum = kShort ? 0.0f : acc[t];
#pragma unroll
                                for (int e = 0; e < E; e += 4) {
                                    const float4 a4 = *reinterpret_cast<const float4*>(ar + e);
                                    const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                                    for (int i = 0; i < 4; ++i) sum = fmaf(p.round_a ? seq_round_bf16(av[i]) : av[i], wv[e + i], sum);
                                }
                                acc[t] = kShort ? acc[t] + sum : sum;
                            }
                        }
                    }
                }
            };
            // two batches of loads: the next one is in flight while the current one is multiplied
            int k0 = k_lo + lane * E;
            uint4 cur[kInFlight];
            load(cur, k0);
            if (early) after_previous();
            for (; k0 < k_hi; k0 += kStep) {
                uint4 nxt[kInFlight];
                load(nxt, k0 + kStep);
                consume(cur, k0);
#pragma unroll
                for (int j = 0; j < kInFlight; ++j) cur[j] = nxt[j];
            }
        } else {
            for (int k = k_lo + lane; k < k_hi; k += 32) {
                const size_t wi = (size_t)wb * p.w_bs + (size_t)n * p.ldw + k;
                const float wv = WD == SLLM_BF16 ? seq_ld(reinterpret_cast<const uint16_t*>(p.W), wi) : reinterpret_cast<const float*>(p.W)[wi];
#pragma unroll
                for (int t = 0; t < kRowsMax; ++t)
                    if (t < p.T) {
                        const float a = A[(size_t)t * p.lda + k];
                        acc[t] = fmaf(p.round_a ? seq_round_bf16(a) : a, wv, acc[t]);
                    }
            }
        }
    } else if (early) {
        after_previous();
    }
#pragma unroll
    for (int t = 0; t < kRowsMax; ++t) {
        const float sum = warp_sum(acc[t]);
        if (lane == 0) part_sum[warp][t] = sum;
    }
    __syncthreads();
    if (part == 0 && n < p.N && lane < p.T) {
        float sum = 0.0f;
        for (int j = 0; j < wpr; ++j) sum += part_sum[warp + j][lane];
        const float v = p.alpha * (sum + (bias ? bias[n] : 0.0f));
        float* c = C + (size_t)lane * p.ldc + n;
        *c = p.accumulate ? *c + v : v;
    }
}

constexpr int kTM = 64, kTN = 64, kTK = 16;

template <int WD>
__global__ void __launch_bounds__(256) seq_linear_tile_kernel(LinArgs p) {
    after_previous();
    __shared__ float As[kTK][kTM + 4];
    __shared__ float Ws[kTK][kTN + 4];
    const int b = blockIdx.z;
    const float* A = p.A + (size_t)b * p.a_bs;
    const float* bias = p.bias ? p.bias + (size_t)b * p.bias_bs : nullptr;
    float* C = p.C + (size_t)b * p.c_bs;
    const int m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
    if (p.rows_dev && m0 >= p.rows_dev[b * p.rows_bs]) return;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lr = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 4;   // loader: row lr of the tile, k columns lk .. lk+3
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < p.K; k0 += kTK) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = k0 + lk + e;
            float a = 0.0f, w = 0.0f;
            if (k < p.K) {
                if (m0 + lr < p.T) {
                    a = A[(size_t)(m0 + lr) * p.lda + k];
                    if (p.round_a) a = seq_round_bf16(a);
                }
                if (n0 + lr < p.N) {
                    const size_t wi = (size_t)b * p.w_bs + (size_t)(n0 + lr) * p.ldw + k;
                    w = WD == SLLM_BF16 ? seq_ld(reinterpret_cast<const uint16_t*>(p.W), wi) : reinterpret_cast<const float*>(p.W)[wi];
                }
            }
            As[lk + e][lr] = a;
            Ws[lk + e][lr] = w;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTK; ++k) {
            const float4 av = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
            const float4 wv = *reinterpret_cast<const float4*>(&Ws[k][tx * 4]);
            const float a4[4] = {av.x, av.y, av.z, av.w}, w4[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a4[i], w4[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= p.T) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= p.N) continue;
            const float v = p.alpha * (acc[i][j] + (bias ? bias[n] : 0.0f));
            float* c = C + (size_t)m * p.ldc + n;
            *c = p.accumulate ? *c + v : v;
        }
    }
}

// A (fp32, row stride lda) -> bf16 [T][K] dense, K a multiple of 8: eight values per thread, 16-byte accesses where A allows them. Bound: HBM. Element by
// element, with a 64-bit division each, 2048 x 2048 took 13.1 us; 5 us like this.
__global__ void __launch_bounds__(256) seq_to_bf16_kernel(const float* A, int lda, uint16_t* out, int T, int K, int vec) {
    after_previous();
    const int per_row = K / 8;
    const long long n = (long long)T * per_row, stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int t = (int)(i / per_row), c = (int)(i - (long long)t * per_row) * 8;
        const float* src = A + (size_t)t * lda + c;
        float4 x, y;
        if (vec) {
            x = *reinterpret_cast<const float4*>(src);
            y = *reinterpret_cast<const float4*>(src + 4);
        } else {
            x = make_float4(src[0], src[1], src[2], src[3]);
            y = make_float4(src[4], src[5], src[6], src[7]);
        }
        auto two = [](float lo, float hi) { return (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16); };
        *reinterpret_cast<uint4*>(out + (size_t)i * 8) = make_uint4(two(x.x, x.y), two(x.z, x.w), two(y.x, y.y), two(y.z, y.w));
    }
}

// C = alpha * (P + bias) (+ C) where P [T][N] dense holds the plain product
__global__ void seq_linear_epilogue_kernel(const float* P, const float* bias, float* C, int ldc, int T, int N,
                                           float alpha, int accumulate) {
    after_previous();
    const size_t n = (size_t)T * N;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / N, j = i % N;
        const float v = alpha * (P[i] + (bias ? bias[j] : 0.0f));
        float* c = C + t * ldc + j;
        *c = accumulate ? *c + v : v;
    }
}

}  // namespace sllm

using namespace sllm;

template <int WD, int TT>
static int launch_rows_body(const sllm::LinArgs& p, int batch, cudaStream_t st) {
    using namespace sllm;
    using Shape = RowsShape<TT>;
    constexpr int E = WD == SLLM_BF16 ? 8 : 4;
    int wk_log2 = 0;      // as many warps along K as one panel of it needs
    while ((1 << wk_log2) < Shape::kWarps && (32 * Shape::kChunks << wk_log2) < p.K / E) ++wk_log2;
    const size_t smem = Shape::kRing + 2 * ((size_t)kRowsBlock * TT * sizeof(float) << wk_log2);
    static bool sized = false;
    if (!sized) {
        SLLM_CUDA(cudaFuncSetAttribute(seq_linear_rows_kernel<WD, TT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       Shape::kRing + 2 * Shape::kWarps * kRowsBlock * TT * (int)sizeof(float)));
        sized = true;
    }
    const dim3 grid(std::max(1, std::min(p.N, sm_count() / batch)), batch);      // one CTA per SM, however many products share the launch
    overlapping(seq_linear_rows_kernel<WD, TT>)<<<grid, Shape::kWarps * 32, smem, st>>>(p, wk_log2);
    return SLLM_OK;
}

static int launch_rows_mma(const sllm::LinArgs& p, int batch, cudaStream_t st) {
    using namespace sllm;
    int wk_log2 = 0;      // as many warps along K as one panel of it needs
    while ((1 << wk_log2) < kMmaWarps && (kMmaSlice << wk_log2) < p.K) ++wk_log2;
    auto smem = [](int wk) { return kMmaWarps * (kMmaRing + kMmaStage) + 2 * ((8 * (mma_block_rows(kMmaWarps >> wk) + 8) * (int)sizeof(float)) << wk); };
    static bool sized = false;
    if (!sized) {
        SLLM_CUDA(cudaFuncSetAttribute(seq_linear_rows_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(4)));
        sized = true;
    }
    const dim3 grid(std::max(1, std::min(p.N, sm_count() / batch)), batch);
    overlapping(seq_linear_rows_mma_kernel)<<<grid, kMmaWarps * 32, smem(wk_log2), st>>>(p, wk_log2);
    return SLLM_OK;
}

// the rows body: up to 8 activation rows per product, `batch` products
static int launch_rows(const sllm::LinArgs& p, int batch, cudaStream_t st) {
    using namespace sllm;
    const bool bf16 = p.w_dtype == SLLM_BF16;
    const int e = bf16 ? 8 : 4;   // elements per 16-byte weight load
    const bool vec = p.K % e == 0 && p.ldw % e == 0 && (p.w_bs % e) == 0 && p.lda % 4 == 0 && (p.a_bs % 4) == 0 && ((uintptr_t)p.W % 16) == 0 &&
                     ((uintptr_t)p.A % 16) == 0;
    // The streaming body needs a few us to start (its ring, its activations, more code). Measured, us, small body | streaming. Up to four rows it is ahead from 1.5 million
    // weights on: 1536 x 1024 bf16 5.2 | 4.2 (one row), 6.1 | 6.0 (three), 6.6 | 6.3 (four), fp32 5.8 | 4.7 and 6.1 | 5.0; 512 x 8192 bf16 5.4 | 5.2 and 8.6 | 7.5; 6144 x
    // 4096 19.4 | 11.4 and 46.9 | 14.6. From five rows on its CTAs hold half the warps and read eight rows of activations each, whatever share of the weights they have.
    // bf16, five rows | eight rows: 2048 x 1024 7.8 | 8.2, 9.5 | 8.7; 512 x 8192 9.7 | 11.9, 13.0 | 12.8; 2800 x 1024 9.5 | 8.8, 12.5 | 9.3; 700 x 8000 16.2 | 13.1, 23.7 | 14.0;
    // 6144 x 4096 85.4 | 21.7 (eight). fp32: 2048 x 1024 7.0 | 7.7, 7.7 | 8.2; 1024 x 4096 9.7 | 11.0, 11.3 | 11.9; 512 x 8192 8.8 | 13.8, 10.2 | 15.7; 600 x 8000 13.6 | 15.2,
    // 18.8 | 16.9; 1000 x 11008 22.0 | 23.4, 26.3 | 26.2; 2800 x 1024 8.6 | 8.4, 9.6 | 8.9; 1500 x 11008 34.0 | 29.0, 43.7 | 32.1. Several products in a launch: 74 of 512 x
    // 512 24 | 9.9 (one row) and 57 | 21 (eight), 80, which leave 68 SMs without one, 26 | 15 and 61 | 33, 160 of 128 x 2048 29 | 24 and 107 | 59.
    const long long rows = (long long)p.N * batch, weights = rows * p.K, sms = sm_count();
    const bool stream = vec && (p.T <= 4          ? weights >= 1500000LL
                                : bf16 ? p.T <= 6 ? weights >= 2800000LL && rows >= 4 * sms : weights >= 2000000LL
                                                  : (weights >= 2800000LL && rows >= 10 * sms) || (p.T >= 7 && weights >= 4500000LL && rows >= 4 * sms));
    // bf16 rows on the tensor cores, where they are ahead of the body that they would take else. That kernel takes 4.3 to 5 us up to some 1.2 million weights (its ring, the split, the last sums),
    // 2 to 3 more where K is longer than one panel, and has tiles that are half empty below four rows an SM; the small body grows with rows times weights. Measured in a captured graph, us, other
    // body | this one, s = the other one streams: two rows 1024 x 1024 3.9 | 4.3, 700 x 2048 5.2 | 4.5, 2048 x 1024 s 5.1 | 5.0, 2048 x 2048 s 5.9 | 6.0; three rows 1024 x 1024 4.3 | 4.4, 700 x 2048 5.7 | 4.6,
    // 400 x 4096 s 5.8 | 5.3, 2048 x 1024 s 6.3 | 5.1; four rows 700 x 1024 3.9 | 4.4, 1024 x 1024 4.6 | 4.4, 256 x 4096 4.7 | 5.3, 400 x 4096 s 6.0 | 5.4, 6144 x 4096 s 14.1 | 13.7, 1024 x 5632 s 8.5 | 8.8; five rows
    // 1500 x 512 4.2 | 4.5, 1024 x 1024 4.9 | 4.5, 256 x 4096 5.2 | 5.5, 512 x 4096 6.4 | 6.0, 512 x 5632 8.1 | 8.4, 256 x 8192 8.5 | 8.6, 512 x 8192 9.7 | 9.0, 140 x 11008 11.6 | 10.3; six rows 400 x 2048 4.5 | 4.9, 512 x 2048
    // 5.1 | 4.9, 400 x 5632 8.2 | 8.4, 512 x 5632 8.9 | 8.5, 64 x 8192 8.5 | 8.1; seven rows 400 x 2048 4.7 | 5.0, 512 x 2048 5.4 | 5.0, 140 x 4096 5.9 | 5.7; eight rows 512 x 1024 4.7 | 4.7, 700 x 1024 5.0 | 4.7, 140 x 4096
    // 6.5 | 5.8, 2048 x 2048 s 11.9 | 6.6, 6144 x 4096 s 23.5 | 14.6, 16384 x 4096 s 46.5 | 27.8. One row is streamed: 6144 x 4096 11.5 | 13.3.
    const bool many = rows >= 4 * sms, one_panel = p.K <= kMmaWarps * kMmaSlice;
    const long long never = LLONG_MAX;
    const long long mma_from = p.T == 2   ? many && one_panel && weights <= 3100000LL ? 1300000LL : never
                               : p.T == 3 ? !one_panel ? never : many ? 1200000LL : 1500000LL
                               : p.T == 4 ? !one_panel ? never : many ? 1000000LL : 1500000LL
                               : p.T == 5 ? many ? 900000LL : p.K > 8192 ? 700000LL : p.K == 8192 ? 3000000LL : one_panel ? 1500000LL : never
                               : p.T == 6 ? many ? 850000LL : p.K >= 8192 ? 500000LL : one_panel ? 1000000LL : 2800000LL
                               : p.T == 7 ? many ? 700000LL : p.K >= 4096 ? 500000LL : 1000000LL
                               : p.T == 8 ? many ? 600000LL : p.K >= 4096 ? 500000LL : 900000LL
                                          : never;
    const bool mma = vec && bf16 && p.round_a && weights >= mma_from;
    if (mma || stream) {
        int rc;
        if (mma) rc = launch_rows_mma(p, batch, st);
        else if (p.T == 1) rc = bf16 ? launch_rows_body<SLLM_BF16, 1>(p, batch, st) : launch_rows_body<SLLM_F32, 1>(p, batch, st);
        else if (p.T == 2) rc = bf16 ? launch_rows_body<SLLM_BF16, 2>(p, batch, st) : launch_rows_body<SLLM_F32, 2>(p, batch, st);
        else if (p.T <= 4) rc = bf16 ? launch_rows_body<SLLM_BF16, 4>(p, batch, st) : launch_rows_body<SLLM_F32, 4>(p, batch, st);
        else rc = bf16 ? launch_rows_body<SLLM_BF16, 8>(p, batch, st) : launch_rows_body<SLLM_F32, 8>(p, batch, st);
        if (rc != SLLM_OK) return rc;
    } else {
        int wpr = 1;   // warps per output column: enough CTAs for ~4 per SM, and no warp with less than 256 weights
        while (wpr < 8 && (long long)p.N * batch * wpr / 8 < 4LL * sm_count() && p.K / (2 * wpr) >= 256) wpr *= 2;
        dim3 grid(((long long)p.N * wpr + 7) / 8, batch);
        const bool brief = weights >= 1500000LL;
        if (bf16 && brief) overlapping(seq_linear_rows_small_kernel<SLLM_BF16, true>)<<<grid, 256, 0, st>>>(p, vec, wpr);
        else if (bf16) overlapping(seq_linear_rows_small_kernel<SLLM_BF16, false>)<<<grid, 256, 0, st>>>(p, vec, wpr);
        else if (brief) overlapping(seq_linear_rows_small_kernel<SLLM_F32, true>)<<<grid, 256, 0, st>>>(p, vec, wpr);
        else overlapping(seq_linear_rows_small_kernel<SLLM_F32, false>)<<<grid, 256, 0, st>>>(p, vec, wpr);
    }
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}

extern "C" int sllm_seq_linear_indexed(const float* A, int32_t lda, int64_t a_bs, int32_t a_div, const void* W, int32_t w_dtype, int32_t ldw, int64_t w_bs,
                                       const int32_t* w_index, float* C, int32_t ldc, int64_t c_bs, int32_t batch, int32_t N, int32_t K, int32_t round_a,
                                       sllm_stream_t stream) {
    using namespace sllm;
    SLLM_REQUIRE(A && W && C && w_index && batch > 0 && batch <= 65535 && N > 0 && K > 0 && a_div >= 1, SLLM_EINVAL, "seq_linear_indexed: bad argument");
    SLLM_REQUIRE(lda >= K && ldw >= K && ldc >= N, SLLM_EINVAL, "seq_linear_indexed: row strides shorter than the rows");
    SLLM_REQUIRE(w_dtype == SLLM_F32 || w_dtype == SLLM_BF16, SLLM_ENOTSUP, "seq_linear_indexed: fp32 or bf16 weights");
    LinArgs p{A, W, nullptr, C, lda, ldw, ldc, 1, N, K, w_dtype, 0, round_a, 1.0f, a_bs, w_bs, 0, c_bs, nullptr, w_index, a_div, 0, 0};
    return launch_rows(p, batch, as_stream(stream));
}

extern "C" int sllm_seq_linear_on_tensor_cores(int32_t T, int32_t N, int32_t K, int32_t w_dtype, int32_t ldw, int32_t batch, int32_t round_a) {
    // bf16 weights and operands, rows that TMA can address (16-byte multiples) and enough work to fill tiles
    return w_dtype == SLLM_BF16 && batch == 1 && round_a && T >= 64 && N >= 64 && K >= 64 && K % 8 == 0 && ldw == K && N % 4 == 0;
}

extern "C" int sllm_seq_linear(const float* A, int32_t lda, const void* W, int32_t w_dtype, int32_t ldw, const float* bias, float* C, int32_t ldc, int32_t T,
                               int32_t N, int32_t K, float alpha, int32_t accumulate, int32_t round_a, int32_t batch, int64_t a_bs, int64_t w_bs,
                               int64_t bias_bs, int64_t c_bs, void* a16, int32_t a16_ready, const int32_t* rows_dev, sllm_stream_t stream) {
    SLLM_REQUIRE(A && W && C && T > 0 && N > 0 && K > 0 && batch >= 1, SLLM_EINVAL, "seq_linear: bad argument");
    SLLM_REQUIRE(lda >= K && ldw >= K && ldc >= N, SLLM_EINVAL, "seq_linear: row strides shorter than the rows");
    SLLM_REQUIRE(w_dtype == SLLM_F32 || w_dtype == SLLM_BF16, SLLM_ENOTSUP, "seq_linear: fp32 or bf16 weights");
    cudaStream_t st = as_stream(stream);
    const int w_fixed = (round_a & SLLM_SEQ_W_FIXED) != 0;
    round_a &= ~SLLM_SEQ_W_FIXED;
    LinArgs p{A, W, bias, C, lda, ldw, ldc, T, N, K, w_dtype, accumulate, round_a, alpha, a_bs, w_bs, bias_bs, c_bs, rows_dev, nullptr, 0, 0, w_fixed};
    if (T <= kRowsMax) return launch_rows(p, batch, st);
    // Steps of 9 to 63 rows: eight at a time through the rows kernels, which read the weights again (from L2, where they fit) but not at a 64 x 64 tile's 78 us per 1024 columns. Measured in a
    // captured graph, us, tiles | eight at a time: 9 rows 512 x 1024 77 | 8.8, 6144 x 4096 342 | 25; 32 rows 512 x 512 41 | 18, 2048 x 2048 178 | 23; 63 rows 512 x 512 43 | 36, 6144 x
    // 4096 371 | 97; with 256 columns 9 rows 21 | 8.6, 32 rows 21 | 18, 48 rows 22 | 27.
    if (T < 64 && w_dtype == SLLM_BF16 && round_a && !rows_dev && batch <= sm_count() && K >= 64 * ((T + kRowsMax - 1) / kRowsMax) && K % 8 == 0 && ldw % 8 == 0 && w_bs % 8 == 0 &&
        lda % 4 == 0 && a_bs % 4 == 0 && ((uintptr_t)W % 16) == 0 && ((uintptr_t)A % 16) == 0) {
        for (int t = 0; t < T; t += kRowsMax) {
            LinArgs q = p;
            q.A += (size_t)t * lda;
            q.C += (size_t)t * ldc;
            q.T = std::min(kRowsMax, T - t);
            if (int rc = launch_rows(q, batch, st)) return rc;
        }
        return SLLM_OK;
    }
    // tensor cores: bf16 weights, a dense bf16 copy of A, rows that TMA can address (16-byte multiples) and enough work to fill tiles
    const bool tensor_cores = a16 && sllm_seq_linear_on_tensor_cores(T, N, K, w_dtype, ldw, batch, round_a) && ((uintptr_t)W % 16) == 0;
    SLLM_REQUIRE(!tensor_cores || !a16_ready || ((uintptr_t)a16 % 16) == 0, SLLM_EINVAL, "seq_linear: bf16 rows that do not start at a multiple of 16 bytes");
    if (tensor_cores && ((uintptr_t)a16 % 16) == 0) {
        static PfCache* cache = pf_cache_create();
        if (!a16_ready) {   // else the kernel that produced A has left its bf16 rows in a16 already
            const size_t n = (size_t)T * K / 8;
            const int vec = lda % 4 == 0 && ((uintptr_t)A % 16) == 0;
            overlapping(seq_to_bf16_kernel)<<<(int)std::min<size_t>((n + 255) / 256, (size_t)sm_count() * 8), 256, 0, st>>>(A, lda, reinterpret_cast<uint16_t*>(a16), T, K, vec);
            ++g_launches;
            SLLM_LAUNCH_CHECK();
        }
        PfGemmArgs a{};
        a.A = a16; a.W = W; a.T = T; a.N = N; a.K = K; a.tiled = 0; a.bn = 0; a.n_valid = N; a.rows_dev = rows_dev;
        if (alpha == 1.0f && ((uintptr_t)C % 16) == 0) {
            // nothing but the bias to do after the product: the GEMM's own epilogue adds it and stores (or adds) straight into C
            a.bias = bias;
            a.epilogue = accumulate ? PF_EPI_RESID : PF_EPI_STORE; a.out = C; a.ld_out = ldc;
            return pf_gemm(cache, a, st);
        }
        float* P = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(a16) + (((size_t)T * K * 2 + 255) / 256) * 256);   // product scratch behind the bf16 rows
        a.epilogue = PF_EPI_STORE; a.out = P; a.ld_out = N;
        const int rc = pf_gemm(cache, a, st);
        if (rc != SLLM_OK) return rc;
        const size_t m = (size_t)T * N;
        overlapping(seq_linear_epilogue_kernel)<<<(int)std::min<size_t>((m + 255) / 256, (size_t)sm_count() * 8), 256, 0, st>>>(P, bias, C, ldc, T, N, alpha, accumulate);
        ++g_launches;
        SLLM_LAUNCH_CHECK_ONLY();
        return SLLM_OK;
    }
    dim3 grid((N + kTN - 1) / kTN, (T + kTM - 1) / kTM, batch);
    if (w_dtype == SLLM_BF16) overlapping_alone(seq_linear_tile_kernel<SLLM_BF16>)<<<grid, 256, 0, st>>>(p);
    else overlapping_alone(seq_linear_tile_kernel<SLLM_F32>)<<<grid, 256, 0, st>>>(p);
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}

extern "C" int sllm_seq_linear_grouped(const void* A, int32_t a_bf16, const void* W, int32_t w_dtype, float* C, const int32_t* counts, int32_t groups, int32_t cap,
                                       int32_t rows_hint, int32_t N, int32_t K, sllm_stream_t stream) {
    SLLM_REQUIRE(A && W && C && counts && groups > 0 && cap > 0 && N > 0 && K > 0, SLLM_EINVAL, "seq_linear_grouped: bad argument");
    SLLM_REQUIRE(w_dtype == SLLM_F32 || w_dtype == SLLM_BF16, SLLM_ENOTSUP, "seq_linear_grouped: fp32 or bf16 weights");
    SLLM_REQUIRE(groups <= 65535, SLLM_ENOTSUP, "seq_linear_grouped: %d groups", groups);
    cudaStream_t st = as_stream(stream);
    if (a_bf16) {        // bf16 rows: ONE tensor-core launch that walks every group's row tiles
        SLLM_REQUIRE(w_dtype == SLLM_BF16 && K % 8 == 0 && K >= 64 && N >= 64 && N % 4 == 0 && ((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0, SLLM_ENOTSUP,
                     "seq_linear_grouped: %d x %d does not fit the tensor-core tiles", N, K);
        SLLM_REQUIRE((long long)groups * cap < 0x7fffffffLL && (long long)groups * N < 0x7fffffffLL, SLLM_ENOTSUP, "seq_linear_grouped: too many rows");
        static PfCache* cache = pf_cache_create();
        PfGemmArgs a{};
        a.A = A; a.W = W; a.T = cap; a.N = N; a.K = K; a.epilogue = PF_EPI_STORE; a.out = C; a.ld_out = N; a.n_valid = N; a.rows_dev = counts;
        a.groups = groups; a.rows_hint = rows_hint;
        return pf_gemm(cache, a, st);
    }
    LinArgs p{(const float*)A, W, nullptr, C, K, K, N, cap, N, K, w_dtype, 0, w_dtype == SLLM_BF16, 1.0f, (long long)cap * K, (long long)N * K, 0, (long long)cap * N,
              counts, nullptr, 0, 1, 0};
    dim3 grid((N + kTN - 1) / kTN, (cap + kTM - 1) / kTM, groups);
    if (w_dtype == SLLM_BF16) overlapping_alone(seq_linear_tile_kernel<SLLM_BF16>)<<<grid, 256, 0, st>>>(p);
    else overlapping_alone(seq_linear_tile_kernel<SLLM_F32>)<<<grid, 256, 0, st>>>(p);
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}
