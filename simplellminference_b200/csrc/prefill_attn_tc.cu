// csrc/prefill_attn_tc.cu — causal attention for a block of T prompt positions on the 5th-generation tensor cores (bf16 cache).
//
// Same work as pf_attn_kernel (prefill_attn.cu; reference source/kernel/cpu/mha_kernel.cpp:36-77): query t at position pos0 + t attends to cache rows
// 0 .. pos0 + t of its kv head; operands bf16, scores, softmax and sums fp32, weights rounded to bf16 for the second product. One CTA per SM, up to TWO
// tiles of 128 queries that share every key and value tile (two query heads of one kv head at the same positions; without such pairs two
// neighbouring query tiles of one head): while one tile's softmax runs, the other's products do. Roles:
//   warp 0 (one lane)   TMA producer: query tiles once, then key and value tiles of 128 positions into rings (128B swizzle; positions beyond the
//                       prompt lie outside the tensor map and read as zeros);
//   warp 1 (one lane)   MMA issuer: S = Q K^T (both K-major) into TMEM; O += P V with P read from TMEM, V as the MN-major operand as it lies;
//   warps 4-7, 8-11     softmax of tile 0 / 1, a thread per query row: tcgen05.ld the scores (once for the maximum, the second half once more for the
//                       weights), exponentials in powers of two, weights packed as bf16 over the scores' own TMEM columns; two values per instruction
//                       where there is one (fma, add), three in the maximum;
//   warps 12-15         O of both tiles: stays in TMEM and is rescaled whenever the maximum of one of the rows of a warp has grown, while the softmax
//                       warps take their exponentials. The reference is the maximum so far: a row's largest weights, which decide its error, are
//                       rounded to bf16 next to 1, where they lose least, and their sum is that of the rounded ones. (With a reference that lagged by up
//                       to 2^8 and the sum of the unrounded ones the result was off by 2.34e-3 instead of 2.29e-3 on the case below and by 2.12e-3 instead
//                       of 1.72e-3 with scores four times as wide; mma.sync 2.29e-3 and 1.73e-3.)
// TMEM: S0 | S1 | O0 | O1, 128 columns each. Bound: the tensor pipe and the exponentials, 1024 clocks each per 128 x 128 tile at head_dim 128, and the chain
// scores -> softmax -> product of a tile; mma.sync, which it replaces for bf16 caches, spent them one after the other in the same warps. Measured, 2048
// queries behind 6144 positions, 32 heads over 8 of 128: 292 us, 822 TFLOP/s (mma.sync 1061 us, 227; rescaling in the softmax warps, one body for masked and other
// tiles and one value per instruction 391; descriptors made anew for every product 315); 256 CTAs on 148 SMs leave a last wave of 108.
#include <type_traits>

#include "prefill.cuh"
#include "tcgen05.cuh"

namespace sllm {
extern int g_tune_pf_pdl;

constexpr int kTaThreads = 512, kTaTile = 128;      // queries of a tile = keys of a tile
constexpr uint32_t kTaTmem = 512;

template <int HD>
struct TaShape {
    static constexpr int kBlocks = HD / 64;                                   // 64-column blocks (128-byte rows) of a tile
    static constexpr int kBlockBytes = kTaTile * 128, kTileBytes = kBlocks * kBlockBytes;
    static constexpr int kStages = HD == 128 ? 2 : 4;
    static constexpr int kSmem = 1024 + (2 + 2 * kStages) * kTileBytes + 512 + 2 * kTaTile * (int)sizeof(float);
};

struct TaArgs {
    uint16_t* out;
    int T, pos0, ldq, heads, group, pair_heads;     // pair_heads: a CTA's two tiles are two heads of a kv head; else two query tiles of one head
    int tiles, items;                               // query tiles of the prompt; tiles of a CTA (1 or 2)
    float scale_log2;
    int32_t* status; unsigned polls;                // where a wait that was given up is reported, and after how many polls it is
};

template <int HD>
__global__ void __launch_bounds__(kTaThreads, 1) pf_attn_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                   const __grid_constant__ CUtensorMap tmV, const TaArgs p) {
    using Sh = TaShape<HD>;
    constexpr int ST = Sh::kStages;
    extern __shared__ uint8_t ta_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ta_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sK = smem;
    uint8_t* sV = sK + ST * Sh::kTileBytes;
    uint8_t* sQ = sV + ST * Sh::kTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sQ + 2 * Sh::kTileBytes);
    uint64_t *kfull = bars, *kempty = kfull + ST, *vfull = kempty + ST, *vempty = vfull + ST, *qfull = vempty + ST;
    // per tile: scores written / factors for O written / weights written and O rescaled / product with the values done
    uint64_t *sfull = qfull + 1, *factors = sfull + 2, *pready = factors + 2, *odone = pready + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(odone + 2);
    float* factor = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 512);       // [2][kTaTile]
    volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // this CTA's tiles: (head, first query) and the key tiles each has to see; the longest first
    const int bx = (int)gridDim.x - 1 - (int)blockIdx.x;
    int head[2], t0[2], nkt[2], items = p.items;       // (every loop over the tiles is unrolled: an index that is not a constant would put these into local memory)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        head[j] = p.items == 2 && p.pair_heads ? 2 * (int)blockIdx.y + j : (int)blockIdx.y;
        const int tile = p.items == 2 && !p.pair_heads ? 2 * bx + j : bx;
        t0[j] = tile * kTaTile;
        nkt[j] = (p.pos0 + min(p.T, t0[j] + kTaTile) + kTaTile - 1) / kTaTile;
        if (j == 1 && (p.items < 2 || tile >= p.tiles)) items = 1;
    }
    if (items == 1) nkt[1] = 0;
    const int kvh = head[0] / p.group, kts = max(nkt[0], nkt[1]);

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        for (int i = 0; i < ST; ++i) { mb_init(kfull + i, 1); mb_init(kempty + i, 1); mb_init(vfull + i, 1); mb_init(vempty + i, 1); }
        mb_init(qfull, 1);
        for (int j = 0; j < 2; ++j) { mb_init(sfull + j, 1); mb_init(factors + j, 128); mb_init(pready + j, 256); mb_init(odone + j, 1); }
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc_alloc(tmem_slot, kTaTmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();

    if (warp == 0) {
        if (elect_one()) {   // ===== TMA producer =====
            mb_expect(qfull, (uint32_t)(items * Sh::kTileBytes));
#pragma unroll
            for (int j = 0; j < 2; ++j)
                for (int c = 0; j < items && c < Sh::kBlocks; ++c) tma_load_2d(sQ + j * Sh::kTileBytes + c * Sh::kBlockBytes, &tmQ, head[j] * HD + 64 * c, t0[j], qfull);
            for (int kt = 0; kt < kts; ++kt) {
                const int s = kt % ST;
                const uint32_t ph = (uint32_t)(kt / ST) & 1;
                if (!tc_wait(kempty + s, ph ^ 1, gave_up, p.polls)) break;
                mb_expect(kfull + s, Sh::kTileBytes);
                for (int c = 0; c < Sh::kBlocks; ++c) tma_load_3d(sK + s * Sh::kTileBytes + c * Sh::kBlockBytes, &tmK, 64 * c, kt * kTaTile, kvh, kfull + s);
                if (!tc_wait(vempty + s, ph ^ 1, gave_up, p.polls)) break;
                mb_expect(vfull + s, Sh::kTileBytes);
                for (int c = 0; c < Sh::kBlocks; ++c) tma_load_3d(sV + s * Sh::kTileBytes + c * Sh::kBlockBytes, &tmV, 64 * c, kt * kTaTile, kvh, vfull + s);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {   // ===== MMA issuer: with descriptors at hand (made anew for each product they took 60 clocks apiece, as long as the product itself) =====
            const uint64_t q_desc = umma_desc_sw128(sQ), k_desc = umma_desc_sw128(sK), v_desc = umma_desc_mn_sw128(sV, Sh::kBlockBytes);      // + bytes / 16: another place
            constexpr uint32_t idesc_s = umma_idesc_bf16(kTaTile, kTaTile), idesc_o = umma_idesc_bf16(kTaTile, HD) | (1u << 16);      // B MN-major
            auto scores = [&](int j, int kt) {
                const uint64_t q = q_desc + (uint32_t)j * (Sh::kTileBytes / 16), k = k_desc + (uint32_t)(kt % ST) * (Sh::kTileBytes / 16);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks) {
                    const uint32_t at = (ks / 4) * (Sh::kBlockBytes / 16) + 2 * (ks % 4);
                    tc_mma_bf16(tmem + 128 * j, q + at, k + at, idesc_s, ks != 0);
                }
                tc_commit(sfull + j);
            };
            auto values = [&](int j, int kt) {
                const uint64_t v = v_desc + (uint32_t)(kt % ST) * (Sh::kTileBytes / 16);
#pragma unroll
                for (int ks = 0; ks < kTaTile / 16; ++ks)
                    tc_mma_bf16_ts(tmem + 256 + 128 * j, tmem + 128 * j + 8 * ks, v + (uint32_t)(ks * 128), idesc_o, (kt | ks) != 0);
                tc_commit(odone + j);
            };
            bool ok = tc_wait(qfull, 0, gave_up, p.polls) && tc_wait(kfull, 0, gave_up, p.polls);
            if (ok) {
                tc_fence_after();
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (j < items) scores(j, 0);
                tc_commit(kempty);
            }
            for (int kt = 0; ok && kt < kts; ++kt) {
                ok = tc_wait(vfull + kt % ST, (uint32_t)(kt / ST) & 1, gave_up, p.polls);
                bool keys = false;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (!ok || kt >= nkt[j]) continue;       // (a CTA's second tile has no key tiles where there is none)
                    ok = tc_wait(pready + j, (uint32_t)kt & 1, gave_up, p.polls);
                    if (!ok) continue;
                    tc_fence_after();
                    values(j, kt);
                    if (kt + 1 >= nkt[j]) continue;
                    if (!keys) {
                        ok = tc_wait(kfull + (kt + 1) % ST, (uint32_t)((kt + 1) / ST) & 1, gave_up, p.polls);
                        keys = true;
                    }
                    // the next scores land where the weights lie that this product is still reading
                    ok = ok && tc_wait(odone + j, (uint32_t)kt & 1, gave_up, p.polls);
                    if (!ok) continue;
                    tc_fence_after();
                    scores(j, kt + 1);
                }
                if (!ok) break;
                tc_commit(vempty + kt % ST);
                if (kt + 1 < kts) tc_commit(kempty + (kt + 1) % ST);
            }
        }
    } else if (warp >= 12) {   // ===== O of both tiles: rescaled while the softmax warps take their exponentials =====
        const int quad = warp & 3, row = quad * 32 + lane;
        bool ok = true;
        for (int kt = 0; ok && kt < kts; ++kt)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (!ok || kt >= nkt[j]) continue;
                ok = tc_wait_warp(factors + j, (uint32_t)kt & 1, gave_up, p.polls);
                if (ok && kt > 0) ok = tc_wait_warp(odone + j, (uint32_t)(kt - 1) & 1, gave_up, p.polls);     // long since: the scores follow that product
                if (!ok) continue;
                tc_fence_after();
                const float f = factor[j * kTaTile + row];
                if (kt > 0 && __any_sync(0xffffffffu, f != 1.0f)) {
                    const uint32_t o_tmem = tmem + ((uint32_t)(quad * 32) << 16) + 256 + 128 * j;
                    const uint64_t ff = tc_two(__float_as_uint(f), __float_as_uint(f));
#pragma unroll 1
                    for (int c = 0; c < HD; c += 64) {
                        uint32_t o[2][32];
                        tc_ld32_async(o_tmem + c, o[0]);
                        tc_ld32_async(o_tmem + c + 32, o[1]);
                        tc_arrived(o[0]);
                        tc_arrived(o[1]);
#pragma unroll
                        for (int i = 0; i < 64; i += 2) {
                            float x, y;
                            tc_split(tc_mul2(tc_two(o[i / 32][i % 32], o[i / 32][i % 32 + 1]), ff), x, y);
                            o[i / 32][i % 32] = __float_as_uint(x);
                            o[i / 32][i % 32 + 1] = __float_as_uint(y);
                        }
                        tc_st32(o_tmem + c, o[0]);
                        tc_st32(o_tmem + c + 32, o[1]);
                    }
                    tc_wait_st();
                }
                tc_fence_before();
                mb_arrive(pready + j);
            }
    } else if (warp >= 4) {   // ===== softmax: TMEM lane quadrant = warp % 4 =====
        const int j = (warp - 4) >> 2, quad = warp & 3, row = quad * 32 + lane, my_t0 = j ? t0[1] : t0[0], my_nkt = j ? nkt[1] : nkt[0], my_head = j ? head[1] : head[0];
        if (j < items) {
            const uint32_t lanes = (uint32_t)(quad * 32) << 16, s_tmem = tmem + lanes + 128 * j, o_tmem = tmem + lanes + 256 + 128 * j;
            const int t = my_t0 + row, qpos = p.pos0 + t, first_pos = p.pos0 + my_t0 + quad * 32;
            const uint64_t scale2 = tc_two(__float_as_uint(p.scale_log2), __float_as_uint(p.scale_log2));
            float ref = -INFINITY, l = 0.0f;            // what the weights are relative to (log2 units); their sum
            bool ok = true;
            // One tile of scores. kMasked: some row of this warp does not see every key of it (columns 0 .. seen are visible); in a body of its own, since
            // comparing and choosing cost as much as everything else a score needs (1700 issue slots a warp and tile, 800 without)
            auto step = [&](auto masked, int kt) {
                constexpr bool kMasked = decltype(masked)::value;
                const int seen = qpos - kt * kTaTile;
                uint32_t a[32], b[32];
                tc_ld32_async(s_tmem + 64, a);
                tc_ld32_async(s_tmem + 96, b);
                tc_arrived(a);
                tc_arrived(b);
                float m0 = -INFINITY, m1 = -INFINITY;
                auto top = [&](const uint32_t* v, int c0) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        float x[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) x[e] = !kMasked || c0 + i + e <= seen ? __uint_as_float(v[i + e]) : -INFINITY;
                        m0 = tc_max3(m0, x[0], x[1]);
                        m1 = tc_max3(m1, x[2], x[3]);
                    }
                };
                top(a, 64);
                top(b, 96);
                tc_ld32_async(s_tmem, a);
                tc_ld32_async(s_tmem + 32, b);
                tc_arrived(a);
                tc_arrived(b);
                top(a, 0);
                top(b, 32);
                const float nr = fmaxf(ref, fmaxf(m0, m1) * p.scale_log2), f = kt == 0 || nr == ref ? 1.0f : tc_exp2(ref - nr);
                factor[j * kTaTile + row] = f;
                mb_arrive(factors + j);
                l *= f;
                ref = nr;
                const uint64_t neg2 = tc_two(__float_as_uint(-ref), __float_as_uint(-ref));
                uint64_t sum0 = 0, sum1 = 0;                                      // (0, 0)
                auto weigh = [&](const uint32_t* v, int c0) {                     // 32 scores -> 16 columns of weights
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float x, y;
                        tc_split(tc_fma2(tc_two(v[i], v[i + 1]), scale2, neg2), x, y);
                        x = tc_exp2(x);
                        y = tc_exp2(y);
                        if (kMasked) {
                            x = c0 + i <= seen ? x : 0.0f;
                            y = c0 + i + 1 <= seen ? y : 0.0f;
                        }
                        w[i / 2] = tc_pack(x, y);
                        uint64_t& sum = (i & 2) ? sum1 : sum0;
                        sum = tc_add2(sum, tc_two(w[i / 2] << 16, w[i / 2] & 0xffff0000u));      // the weights as they are used
                    }
                    tc_st16(s_tmem + c0 / 2, w);
                };
                weigh(a, 0);
                weigh(b, 32);
                tc_ld32_async(s_tmem + 64, a);
                tc_ld32_async(s_tmem + 96, b);
                tc_arrived(a);
                tc_arrived(b);
                weigh(a, 64);
                weigh(b, 96);
                float l0, l1;
                tc_split(tc_add2(sum0, sum1), l0, l1);
                l += l0 + l1;
            };
            for (int kt = 0; kt < my_nkt; ++kt) {
                ok = tc_wait_warp(sfull + j, (uint32_t)kt & 1, gave_up, p.polls);
                if (!ok) break;
                tc_fence_after();
                if (kt * kTaTile + kTaTile - 1 > first_pos) step(std::true_type{}, kt);
                else step(std::false_type{}, kt);
                tc_wait_st();
                tc_fence_before();
                mb_arrive(pready + j);
            }
            ok = ok && tc_wait_warp(odone + j, (uint32_t)(my_nkt - 1) & 1, gave_up, p.polls);
            tc_fence_after();
            const float inv = 1.0f / l;
#pragma unroll 1
            for (int c = 0; ok && c < HD; c += 32) {
                uint32_t o[32];
                tc_ld32_async(o_tmem + c, o);
                tc_arrived(o);
                if (t < p.T) {
                    uint4* dst = reinterpret_cast<uint4*>(p.out + (size_t)t * p.ldq + (size_t)my_head * HD + c);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        auto two = [&](int e) { return tc_pack(__uint_as_float(o[8 * i + e]) * inv, __uint_as_float(o[8 * i + e + 1]) * inv); };
                        dst[i] = make_uint4(two(0), two(2), two(4), two(6));
                    }
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*gave_up) tc_gave_up(p.status);
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc(tmem, kTaTmem);
    }
}

template <int HD>
static int ta_launch(const uint16_t* q, const void* kc, const void* vc, uint16_t* out, int T, int pos0, int S, int heads, int kv_heads, cudaStream_t st) {
    using Sh = TaShape<HD>;
    static bool configured = false;
    if (!configured) {
        SLLM_CUDA(cudaFuncSetAttribute(pf_attn_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
        configured = true;
    }
    CUtensorMap tmQ, tmK, tmV;
    {
        const cuuint64_t dims[2] = {(cuuint64_t)heads * HD, (cuuint64_t)T};
        const cuuint64_t strides[1] = {(cuuint64_t)heads * HD * 2};
        const cuuint32_t box[2] = {64, kTaTile};
        if (int rc = tc_encode_bf16(&tmQ, q, 2, dims, strides, box)) return rc;
    }
    const cuuint64_t dims[3] = {HD, (cuuint64_t)(pos0 + T), (cuuint64_t)kv_heads};      // positions beyond the prompt read as zeros
    const cuuint64_t strides[2] = {HD * 2, (cuuint64_t)S * HD * 2};
    const cuuint32_t box[3] = {64, kTaTile, 1};
    if (int rc = tc_encode_bf16(&tmK, kc, 3, dims, strides, box)) return rc;
    if (int rc = tc_encode_bf16(&tmV, vc, 3, dims, strides, box)) return rc;
    TaArgs a{};
    a.out = out; a.T = T; a.pos0 = pos0; a.ldq = heads * HD; a.heads = heads; a.group = heads / kv_heads;
    a.pair_heads = a.group % 2 == 0;
    a.tiles = (T + kTaTile - 1) / kTaTile;
    // two tiles per CTA hide each other's softmax and share their loads, unless single ones would still leave SMs idle
    a.items = (long long)a.tiles * heads > sm_count() ? 2 : 1;
    if (int rc = status_check()) return rc;
    if (int rc = status_word(&a.status)) return rc;
    a.polls = (unsigned)g_tune_tc_polls;
    a.scale_log2 = (1.0f / sqrtf((float)HD)) * 1.4426950408889634f;
    const dim3 grid(a.items == 2 && !a.pair_heads ? (a.tiles + 1) / 2 : a.tiles, a.items == 2 && a.pair_heads ? heads / 2 : heads);
    LaunchCfg lc(grid, dim3(kTaThreads), Sh::kSmem, st, g_tune_pf_pdl != 0);
    SLLM_CUDA(cudaLaunchKernelEx(&lc.cfg, pf_attn_tc_kernel<HD>, tmQ, tmK, tmV, a));
    g_launches++;
    SLLM_LAUNCH_CHECK_ONLY();
    return SLLM_OK;
}

int pf_attention_tc(const uint16_t* q, const void* kc, const void* vc, uint16_t* out, int T, int pos0, int S, int hd, int heads, int kv_heads, cudaStream_t st) {
    return hd == 128 ? ta_launch<128>(q, kc, vc, out, T, pos0, S, heads, kv_heads, st) : ta_launch<64>(q, kc, vc, out, T, pos0, S, heads, kv_heads, st);
}

}  // namespace sllm
