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
// queries behind 6144 positions, 32 heads over 8 of 128: 287 us with a CTA per work item, 245 us and 980 TFLOP/s with equal shares (below); under the power limit, calls
// without a pause for half a second, 292 and 274 (mma.sync 1061 us; rescaling in the softmax warps, one body for masked and other tiles and one value per instruction 391;
// descriptors made anew for every product 315).
//
// Shares. A CTA per work item leaves the last wave half empty (256 items on 148 SMs) and most SMs without work where there are few queries behind a long context. With
// scratch the key tiles of all items form one row that is cut into equal runs, one a CTA, which goes through its run item by item: barriers and TMEM are set up once, and
// the next item's queries load while the last one's weights are taken. The items that a cut goes through (one or two a CTA) leave O, reference and sum as fp32 parts, which
// ta_merge_kernel adds. Measured, us, CTA per item | shares, heads of 128: 2048 queries from the start, 32 heads 71 | 64, 512 behind 2000 47 | 38, 1500 behind 3000, 16 heads
// 88 | 64, 256 behind 5000, 8 heads 89 | 33, 100 behind 6000, 32 heads over 2 101 | 32, 300 behind 4000, 24 heads 74 | 40; heads of 64 (mma.sync | shares): 256 behind 2000, 32
// heads 42 | 23, 1000 behind 5000, 8 heads 106 | 37, 100 behind 1000, 8 heads 22 | 14, 300 behind 4000, 24 heads 77 | 37.
#include <type_traits>

#include "prefill.cuh"
#include "tcgen05.cuh"

namespace sllm {
extern int g_tune_pf_pdl;

constexpr int kTaThreads = 512, kTaTile = 128;      // queries of a tile = keys of a tile
constexpr uint32_t kTaTmem = 512;
// What ta_plan reckons with, in times of a key tile of two query tiles (2.2 us): a key tile of a single query tile; the parts' way to the scratch, their merge and its launch, at
// heads of 128 and of 64; 128 keys of the mma.sync kernel at heads of 64; and the fewest key tiles that a share is made for. With a merge at 4.5 instead of 5.5 shares were taken
// where they lost (1024 queries from the start, 16 heads of 128: 22.0 | 23.1). Least shares of 2, 3, 4, 6 and 8 tiles: 64 queries behind 2000, 8 heads 20.7, 22.0, 23.9, 23.2 and
// 27.3 us, 256 behind 5000 32.3, 30.3, 28.6, 29.0 and 33.6, one query behind 1000, 32 heads 17.8, 20.8, 18.6, 25.0 and 24.4.
constexpr float kTaSingle = 0.85f, kTaMerge = 5.5f, kTaMerge64 = 6.0f, kTaSync = 1.05f;
constexpr int kTaLeast = 2;

template <int HD>
struct TaShape {
    static constexpr int kBlocks = HD / 64;                                   // 64-column blocks (128-byte rows) of a tile
    static constexpr int kBlockBytes = kTaTile * 128, kTileBytes = kBlocks * kBlockBytes;
    static constexpr int kStages = HD == 128 ? 2 : 4;
    static constexpr int kSmem = 1024 + (2 + 2 * kStages) * kTileBytes + 512 + 2 * kTaTile * (int)sizeof(float);
    // what a CTA leaves of a work item that others have a part of, too: per tile O as [HD / 4][128 rows][4], then the rows' references and sums
    static constexpr int kPartTile = kTaTile * (HD + 2), kPart = 2 * kPartTile;
};

struct TaArgs {
    uint16_t* out;
    int T, pos0, ldq, heads, group, pair_heads;     // pair_heads: a CTA's two tiles are two heads of a kv head; else two query tiles of one head
    int tiles, items;                               // query tiles of the prompt; tiles of a CTA (1 or 2)
    float scale_log2;
    // Shares: key tiles of all work items in a row, [ctas] neighbouring runs of them as equal as can be; a work item = the tiles that a CTA has at a time, `row` of them
    // a head or pair of heads, `row_keys` key tiles together. units = 0: every CTA has one work item, all of it.
    int units, ctas, row, row_keys;
    float* parts;                                   // [2 * ctas][TaShape::kPart]: the first and the last work item of a CTA's share, where it is not all the CTA's
    int32_t* status; unsigned polls;                // where a wait that was given up is reported, and after how many polls it is
};

// first key tile of share c, and the share that key tile u belongs to
__host__ __device__ __forceinline__ int ta_share(int c, int units, int ctas) { return (int)((long long)c * units / ctas); }
__host__ __device__ __forceinline__ int ta_owner(int u, int units, int ctas) { return (int)(((long long)(u + 1) * ctas - 1) / units); }
// key tiles of work item x of its row: those that its last query sees
__host__ __device__ __forceinline__ int ta_keys(int T, int pos0, int queries, int x) {
    const int last = (x + 1) * queries;
    return (pos0 + (last < T ? last : T) + kTaTile - 1) / kTaTile;
}

// A CTA's way through its share: (x, y) = work item and row, k0 .. k1 = its key tiles that are this CTA's. Every role walks it by itself.
template <bool kShares>
struct TaWalk {
    int x, y, k0, k1, left;
    const TaArgs& p;
    int queries;
    __device__ __forceinline__ explicit TaWalk(const TaArgs& args) : p(args), queries(args.items == 2 && !args.pair_heads ? 2 * kTaTile : kTaTile) {
        if constexpr (kShares) {
            const int c = (int)blockIdx.x, first = ta_share(c, p.units, p.ctas);
            left = ta_share(c + 1, p.units, p.ctas) - first;
            y = first / p.row_keys;
            k0 = first % p.row_keys;
            x = 0;
            for (int n; k0 >= (n = ta_keys(p.T, p.pos0, queries, x)); ++x) k0 -= n;
            k1 = min(ta_keys(p.T, p.pos0, queries, x), k0 + left);
        } else {
            x = (int)gridDim.x - 1 - (int)blockIdx.x;      // the longest first
            y = (int)blockIdx.y;
            k0 = 0;
            k1 = left = ta_keys(p.T, p.pos0, queries, x);
        }
    }
    __device__ __forceinline__ bool next() {
        if (!kShares) return false;
        left -= k1 - k0;
        if (left <= 0) return false;
        if (++x == p.row) { x = 0; ++y; }
        k0 = 0;
        k1 = min(ta_keys(p.T, p.pos0, queries, x), left);
        return true;
    }
    __device__ __forceinline__ bool whole() const { return !kShares || (k0 == 0 && k1 == ta_keys(p.T, p.pos0, queries, x)); }
    // tile j: its head, its first query, how many of the key tiles k0 .. k1 it has to see
    __device__ __forceinline__ int head(int j) const { return p.items == 2 && p.pair_heads ? 2 * y + j : y; }
    __device__ __forceinline__ int first(int j) const { return (p.items == 2 && !p.pair_heads ? 2 * x + j : x) * kTaTile; }
    __device__ __forceinline__ bool has(int j) const { return j == 0 || (p.items == 2 && first(1) < p.T); }
    __device__ __forceinline__ int keys(int j) const { return has(j) ? max(0, min(k1, (p.pos0 + min(p.T, first(j) + kTaTile) + kTaTile - 1) / kTaTile) - k0) : 0; }
};

// kShares: CTAs have shares (units > 0). Without them the walk is one work item, and its code 0.2 to 0.3 us less of a short call (100 queries from the start, 32 heads of 128: 6.0 | 6.3).
template <int HD, bool kShares>
__global__ void __launch_bounds__(kTaThreads, 1) pf_attn_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                                                                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ TaArgs p) {
    using Sh = TaShape<HD>;
    constexpr int ST = Sh::kStages;
    extern __shared__ uint8_t ta_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ta_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sK = smem;
    uint8_t* sV = sK + ST * Sh::kTileBytes;
    uint8_t* sQ = sV + ST * Sh::kTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sQ + 2 * Sh::kTileBytes);
    uint64_t *kfull = bars, *kempty = kfull + ST, *vfull = kempty + ST, *vempty = vfull + ST, *qfull = vempty + ST, *qempty = qfull + 1;
    // per tile: scores written / factors for O written / weights written and O rescaled / product with the values done
    uint64_t *sfull = qempty + 1, *factors = sfull + 2, *pready = factors + 2, *odone = pready + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(odone + 2);
    float* factor = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 512);       // [2][kTaTile]
    volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        for (int i = 0; i < ST; ++i) { mb_init(kfull + i, 1); mb_init(kempty + i, 1); mb_init(vfull + i, 1); mb_init(vempty + i, 1); }
        mb_init(qfull, 1);
        mb_init(qempty, 1);
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
            TaWalk<kShares> w(p);
            int g = 0;                                      // key tiles so far
            uint32_t seg = 0;
            bool ok = true;
            do {
                const int kvh = w.head(0) / p.group, n = w.has(1) ? 2 : 1;
                ok = tc_wait(qempty, (seg & 1) ^ 1, gave_up, p.polls);
                if (!ok) break;
                mb_expect(qfull, (uint32_t)(n * Sh::kTileBytes));
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    for (int c = 0; j < n && c < Sh::kBlocks; ++c) tma_load_2d(sQ + j * Sh::kTileBytes + c * Sh::kBlockBytes, &tmQ, w.head(j) * HD + 64 * c, w.first(j), qfull);
                for (int kt = w.k0; kt < w.k1; ++kt, ++g) {
                    const int s = g % ST;
                    const uint32_t ph = (uint32_t)(g / ST) & 1;
                    ok = tc_wait(kempty + s, ph ^ 1, gave_up, p.polls);
                    if (!ok) break;
                    mb_expect(kfull + s, Sh::kTileBytes);
                    for (int c = 0; c < Sh::kBlocks; ++c) tma_load_3d(sK + s * Sh::kTileBytes + c * Sh::kBlockBytes, &tmK, 64 * c, kt * kTaTile, kvh, kfull + s);
                    ok = tc_wait(vempty + s, ph ^ 1, gave_up, p.polls);
                    if (!ok) break;
                    mb_expect(vfull + s, Sh::kTileBytes);
                    for (int c = 0; c < Sh::kBlocks; ++c) tma_load_3d(sV + s * Sh::kTileBytes + c * Sh::kBlockBytes, &tmV, 64 * c, kt * kTaTile, kvh, vfull + s);
                }
                ++seg;
            } while (ok && w.next());
        }
    } else if (warp == 1) {
        if (elect_one()) {   // ===== MMA issuer: with descriptors at hand (made anew for each product they took 60 clocks apiece, as long as the product itself) =====
            const uint64_t q_desc = umma_desc_sw128(sQ), k_desc = umma_desc_sw128(sK), v_desc = umma_desc_mn_sw128(sV, Sh::kBlockBytes);      // + bytes / 16: another place
            constexpr uint32_t idesc_s = umma_idesc_bf16(kTaTile, kTaTile), idesc_o = umma_idesc_bf16(kTaTile, HD) | (1u << 16);      // B MN-major
            auto scores = [&](int j, int g) {
                const uint64_t q = q_desc + (uint32_t)j * (Sh::kTileBytes / 16), k = k_desc + (uint32_t)(g % ST) * (Sh::kTileBytes / 16);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks) {
                    const uint32_t at = (ks / 4) * (Sh::kBlockBytes / 16) + 2 * (ks % 4);
                    tc_mma_bf16(tmem + 128 * j, q + at, k + at, idesc_s, ks != 0);
                }
                tc_commit(sfull + j);
            };
            auto values = [&](int j, int g, bool more) {
                const uint64_t v = v_desc + (uint32_t)(g % ST) * (Sh::kTileBytes / 16);
#pragma unroll
                for (int ks = 0; ks < kTaTile / 16; ++ks)
                    tc_mma_bf16_ts(tmem + 256 + 128 * j, tmem + 128 * j + 8 * ks, v + (uint32_t)(ks * 128), idesc_o, more || ks != 0);
                tc_commit(odone + j);
            };
            TaWalk<kShares> w(p);
            int g = 0;                                      // key tiles so far, and those of them that tile 0 and 1 saw
            uint32_t seg = 0, done[2] = {0, 0};
            bool ok = true;
            do {
                const int n = w.k1 - w.k0, nkt[2] = {w.keys(0), w.keys(1)};
                ok = tc_wait(qfull, seg & 1, gave_up, p.polls) && tc_wait(kfull + g % ST, (uint32_t)(g / ST) & 1, gave_up, p.polls);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (!ok || nkt[j] == 0) continue;
                    // they land where the last weights of the item before lie
                    if (done[j]) ok = tc_wait(odone + j, (done[j] - 1) & 1, gave_up, p.polls);
                    if (!ok) continue;
                    tc_fence_after();
                    scores(j, g);
                }
                if (!ok) break;
                tc_commit(kempty + g % ST);
                if (n == 1) tc_commit(qempty);
                for (int kt = 0; kt < n; ++kt, ++g) {
                    ok = tc_wait(vfull + g % ST, (uint32_t)(g / ST) & 1, gave_up, p.polls);
                    bool keys = false;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (!ok || kt >= nkt[j]) continue;
                        ok = tc_wait(pready + j, done[j] & 1, gave_up, p.polls);
                        if (!ok) continue;
                        tc_fence_after();
                        values(j, g, kt != 0);
                        ++done[j];
                        if (kt + 1 >= nkt[j]) continue;
                        if (!keys) {
                            ok = tc_wait(kfull + (g + 1) % ST, (uint32_t)((g + 1) / ST) & 1, gave_up, p.polls);
                            keys = true;
                        }
                        // the next scores land where the weights lie that this product is still reading
                        ok = ok && tc_wait(odone + j, (done[j] - 1) & 1, gave_up, p.polls);
                        if (!ok) continue;
                        tc_fence_after();
                        scores(j, g + 1);
                    }
                    if (!ok) break;
                    tc_commit(vempty + g % ST);
                    if (kt + 1 < n) tc_commit(kempty + (g + 1) % ST);
                    if (kt + 2 == n) tc_commit(qempty);
                }
                ++seg;
            } while (ok && w.next());
        }
    } else if (warp >= 12) {   // ===== O of both tiles: rescaled while the softmax warps take their exponentials =====
        const int quad = warp & 3, row = quad * 32 + lane;
        TaWalk<kShares> w(p);
        uint32_t done[2] = {0, 0};
        bool ok = true;
        do {
          const int n = w.k1 - w.k0, nkt[2] = {w.keys(0), w.keys(1)};
          for (int kt = 0; ok && kt < n; ++kt)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (!ok || kt >= nkt[j]) continue;
                ok = tc_wait_warp(factors + j, done[j] & 1, gave_up, p.polls);
                if (ok && kt > 0) ok = tc_wait_warp(odone + j, (done[j] - 1) & 1, gave_up, p.polls);     // long since: the scores follow that product
                if (!ok) continue;
                ++done[j];
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
        } while (ok && w.next());
    } else if (warp >= 4) {   // ===== softmax: TMEM lane quadrant = warp % 4 =====
        const int j = (warp - 4) >> 2, quad = warp & 3, row = quad * 32 + lane;
        const uint32_t lanes = (uint32_t)(quad * 32) << 16, s_tmem = tmem + lanes + 128 * j, o_tmem = tmem + lanes + 256 + 128 * j;
        const uint64_t scale2 = tc_two(__float_as_uint(p.scale_log2), __float_as_uint(p.scale_log2));
        TaWalk<kShares> w(p);
        uint32_t done = 0;
        bool ok = true, at_first = true;
        do {
            if (!w.has(j)) { at_first = false; continue; }
            const int n = w.keys(j), t = w.first(j) + row, qpos = p.pos0 + t, first_pos = qpos - lane;
            float ref = -INFINITY, l = 0.0f;            // what the weights are relative to (log2 units); their sum
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
                const float nr = fmaxf(ref, fmaxf(m0, m1) * p.scale_log2), f = kt == w.k0 || nr == ref ? 1.0f : tc_exp2(ref - nr);
                factor[j * kTaTile + row] = f;
                mb_arrive(factors + j);
                l *= f;
                ref = nr;
                // where every score so far is -inf, -inf - ref were no number: relative to 0 their weights are 0 (a share may start with such keys, in the middle of a row that sees others)
                const uint32_t neg = __float_as_uint(ref == -INFINITY ? 0.0f : -ref);
                const uint64_t neg2 = tc_two(neg, neg);
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
            for (int kt = w.k0; kt < w.k0 + n; ++kt) {
                ok = tc_wait_warp(sfull + j, done & 1, gave_up, p.polls);
                if (!ok) break;
                ++done;
                tc_fence_after();
                if (kt * kTaTile + kTaTile - 1 > first_pos) step(std::true_type{}, kt);
                else step(std::false_type{}, kt);
                tc_wait_st();
                tc_fence_before();
                mb_arrive(pready + j);
            }
            if (ok && n > 0) ok = tc_wait_warp(odone + j, (done - 1) & 1, gave_up, p.polls);
            tc_fence_after();
            if (w.whole()) {
                const float inv = 1.0f / l;
#pragma unroll 1
                for (int c = 0; ok && c < HD; c += 32) {
                    uint32_t o[32];
                    tc_ld32_async(o_tmem + c, o);
                    tc_arrived(o);
                    if (t < p.T) {
                        uint4* dst = reinterpret_cast<uint4*>(p.out + (size_t)t * p.ldq + (size_t)w.head(j) * HD + c);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            auto two = [&](int e) { return tc_pack(__uint_as_float(o[8 * i + e]) * inv, __uint_as_float(o[8 * i + e + 1]) * inv); };
                            dst[i] = make_uint4(two(0), two(2), two(4), two(6));
                        }
                    }
                    __syncwarp();
                }
            } else {                                    // the rest of its keys are other CTAs': as it is, to be put together by ta_merge_kernel
                float* part = p.parts + (size_t)(2 * blockIdx.x + (at_first ? 0 : 1)) * Sh::kPart + j * Sh::kPartTile;
#pragma unroll 1
                for (int c = 0; ok && n > 0 && c < HD; c += 32) {
                    uint32_t o[32];
                    tc_ld32_async(o_tmem + c, o);
                    tc_arrived(o);
#pragma unroll
                    for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(part)[(c / 4 + i) * kTaTile + row] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                }
                part[HD * kTaTile + row] = ref;
                part[(HD + 1) * kTaTile + row] = l;
            }
            at_first = false;
        } while (ok && w.next());
    }
    tc_fence_before();
    __syncthreads();
    if (*gave_up) tc_gave_up(p.status);
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc(tmem, kTaTmem);
    }
}

// Work items that lie in several shares: their parts brought to one reference and added. blockIdx: work item, row, tile and kTaMergeCols columns of it; a thread per
// query, whose loads do not wait for one another: with few items in many parts (256 queries, 8 heads, 20 parts each) the reads of one item are a chain otherwise. Bound by
// those reads, up to 39 MB that the L2 mostly has.
template <int HD, int kTaMergeCols>
__global__ void __launch_bounds__(kTaTile) ta_merge_kernel(const TaArgs p) {
    using Sh = TaShape<HD>;
    constexpr int kSplit = HD / kTaMergeCols;
    const int x = blockIdx.x, y = blockIdx.y, j = blockIdx.z / kSplit, c = blockIdx.z % kSplit * kTaMergeCols, row = threadIdx.x;
    const bool pair_tiles = p.items == 2 && !p.pair_heads;
    const int queries = pair_tiles ? 2 * kTaTile : kTaTile, head = pair_tiles ? y : p.items * y + j, t = (pair_tiles ? 2 * x + j : x) * kTaTile + row;
    int from = y * p.row_keys;
    for (int i = 0; i < x; ++i) from += ta_keys(p.T, p.pos0, queries, i);
    const int to = from + ta_keys(p.T, p.pos0, queries, x), c0 = ta_owner(from, p.units, p.ctas), n = ta_owner(to - 1, p.units, p.ctas) - c0;
    pdl_wait();
    pdl_launch_dependents();
    if (n == 0 || t >= p.T) return;
    // a share's first work item is in its first place, and no other of its work items but the last can be in several shares
    const float* rest = p.parts + (size_t)(2 * c0) * Sh::kPart + j * Sh::kPartTile;
    const float* head_part = rest + (ta_share(c0, p.units, p.ctas) < from ? Sh::kPart : 0);
    auto part_of = [&](int s) { return s == 0 ? head_part : rest + (size_t)(2 * s) * Sh::kPart; };
    float top = -INFINITY, sum = 0.0f;
#pragma unroll 8
    for (int s = 0; s <= n; ++s) top = fmaxf(top, __ldcg(part_of(s) + HD * kTaTile + row));
    float o[kTaMergeCols] = {};
#pragma unroll 4
    for (int s = 0; s <= n; ++s) {
        const float* part = part_of(s);
        const float ref = __ldcg(part + HD * kTaTile + row), l = __ldcg(part + (HD + 1) * kTaTile + row);
        const bool none = ref == -INFINITY && l == 0.0f;      // none of its keys is visible to this query; its O may never have been written
        const float f = none ? 0.0f : ref == top ? 1.0f : tc_exp2(ref - top);
        sum = fmaf(l, f, sum);
#pragma unroll
        for (int i = 0; i < kTaMergeCols / 4; ++i) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(part) + (c / 4 + i) * kTaTile + row);
            o[4 * i] = fmaf(none ? 0.0f : v.x, f, o[4 * i]);
            o[4 * i + 1] = fmaf(none ? 0.0f : v.y, f, o[4 * i + 1]);
            o[4 * i + 2] = fmaf(none ? 0.0f : v.z, f, o[4 * i + 2]);
            o[4 * i + 3] = fmaf(none ? 0.0f : v.w, f, o[4 * i + 3]);
        }
    }
    const float inv = 1.0f / sum;
    uint4* dst = reinterpret_cast<uint4*>(p.out + (size_t)t * p.ldq + (size_t)head * HD + c);
#pragma unroll
    for (int i = 0; i < kTaMergeCols / 8; ++i) {
        auto two = [&](int e) { return tc_pack(o[8 * i + e] * inv, o[8 * i + e + 1] * inv); };
        dst[i] = make_uint4(two(0), two(2), two(4), two(6));
    }
}

// How a call is divided: tiles of a CTA at a time, and into how many shares, if any.
struct TaPlan { int items, pair_heads, tiles, row, rows, row_keys, units, ctas; };
static TaPlan ta_plan(int T, int pos0, int hd, int heads, int kv_heads, bool scratch) {
    TaPlan q{};
    const int sms = sm_count();
    q.pair_heads = heads / kv_heads % 2 == 0;
    q.tiles = (T + kTaTile - 1) / kTaTile;
    auto shape = [&](int items) {
        q.items = items;
        const bool pair_tiles = items == 2 && !q.pair_heads;
        q.row = pair_tiles ? (q.tiles + 1) / 2 : q.tiles;
        q.rows = items == 2 && q.pair_heads ? heads / 2 : heads;
        q.row_keys = 0;
        for (int x = 0; x < q.row; ++x) q.row_keys += ta_keys(T, pos0, pair_tiles ? 2 * kTaTile : kTaTile, x);
    };
    // two tiles per CTA hide each other's softmax and share their loads, unless single ones would still leave SMs idle
    const int whole = (long long)q.tiles * heads > sms ? 2 : 1;
    shape(whole);
    if (!scratch) return q;
    const int longest = (pos0 + T + kTaTile - 1) / kTaTile;
    const float whole_cost = pf_attention_fills(T, pos0 + T, hd, heads) ? (float)(((long long)q.row * q.rows + sms - 1) / sms) * longest * (whole == 2 ? 1.0f : kTaSingle)
                                                                        : longest * kTaSync - (kTaMerge64 - kTaMerge);
    shape(q.tiles * heads > 1 && (q.pair_heads || q.tiles > 1) ? 2 : 1);
    const long long units = (long long)q.row_keys * q.rows;
    const int ctas = (int)min((long long)sms, (units + kTaLeast - 1) / kTaLeast);
    const float cost = (float)((units + ctas - 1) / ctas) * (q.items == 2 ? 1.0f : kTaSingle) + kTaMerge;
    if (units < (1 << 30) && cost < whole_cost) {
        q.units = (int)units;
        q.ctas = ctas;
    } else {
        shape(whole);
    }
    return q;
}
size_t pf_attention_tc_scratch(int T, int pos0, int hd, int heads, int kv_heads) {
    const TaPlan q = ta_plan(T, pos0, hd, heads, kv_heads, true);
    return q.units ? (size_t)2 * q.ctas * (hd == 128 ? TaShape<128>::kPart : TaShape<64>::kPart) : 0;
}

template <int HD>
static int ta_launch(const uint16_t* q, const void* kc, const void* vc, uint16_t* out, int T, int pos0, int S, int heads, int kv_heads, float* scratch, cudaStream_t st) {
    using Sh = TaShape<HD>;
    static bool configured = false;
    if (!configured) {
        SLLM_CUDA(cudaFuncSetAttribute(pf_attn_tc_kernel<HD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
        SLLM_CUDA(cudaFuncSetAttribute(pf_attn_tc_kernel<HD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
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
    const TaPlan plan = ta_plan(T, pos0, HD, heads, kv_heads, scratch != nullptr);
    a.pair_heads = plan.pair_heads; a.tiles = plan.tiles; a.items = plan.items;
    a.units = plan.units; a.ctas = plan.ctas; a.row = plan.row; a.row_keys = plan.row_keys; a.parts = scratch;
    if (int rc = status_check()) return rc;
    if (int rc = status_word(&a.status)) return rc;
    a.polls = (unsigned)g_tune_tc_polls;
    a.scale_log2 = (1.0f / sqrtf((float)HD)) * 1.4426950408889634f;
    const dim3 grid(plan.units ? plan.ctas : plan.row, plan.units ? 1 : plan.rows);
    LaunchCfg lc(grid, dim3(kTaThreads), Sh::kSmem, st, g_tune_pf_pdl != 0);
    SLLM_CUDA(cudaLaunchKernelEx(&lc.cfg, plan.units ? pf_attn_tc_kernel<HD, true> : pf_attn_tc_kernel<HD, false>, tmQ, tmK, tmV, a));
    g_launches++;
    if (plan.units) {
        auto merge = [&](auto cols) {
            constexpr int kCols = decltype(cols)::value;
            LaunchCfg lm(dim3(plan.row, plan.rows, (unsigned)(plan.items * (HD / kCols))), dim3(kTaTile), 0, st, g_tune_pf_pdl != 0);
            SLLM_CUDA(cudaLaunchKernelEx(&lm.cfg, ta_merge_kernel<HD, kCols>, a));
            return SLLM_OK;
        };
        // 32 columns a block write whole sectors of the result; with few work items (and then many parts of each) 8 keep more reads on their way. 32 | 8 columns, us a call: 2048
        // queries behind 6144, 32 heads 244 | 249, from the start 64 | 69, but 256 behind 5000, 8 heads 48 | 32 and 100 behind 6000, 32 heads over 2 41 | 32
        const bool many = plan.row * plan.rows * plan.items * (HD / 32) >= 4 * sm_count();
        if (int rc = many ? merge(std::integral_constant<int, 32>{}) : merge(std::integral_constant<int, 8>{})) return rc;
        g_launches++;
    }
    SLLM_LAUNCH_CHECK_ONLY();
    return SLLM_OK;
}

int pf_attention_tc(const uint16_t* q, const void* kc, const void* vc, uint16_t* out, int T, int pos0, int S, int hd, int heads, int kv_heads, float* scratch,
                    cudaStream_t st) {
    return hd == 128 ? ta_launch<128>(q, kc, vc, out, T, pos0, S, heads, kv_heads, scratch, st) : ta_launch<64>(q, kc, vc, out, T, pos0, S, heads, kv_heads, scratch, st);
}

}  // namespace sllm
