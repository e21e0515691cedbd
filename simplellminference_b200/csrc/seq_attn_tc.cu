// csrc/seq_attn_tc.cu — attention of prompt portions over the paged cache on the 5th-generation tensor cores: bf16 pools, key and value heads of 64 or 128.
//
// The tensor-core body of seq_attn.cu keeps a warp's 16 queries in its registers and stages tiles of 32 keys for 64 rows; here 128 rows = the query heads
// of a kv head (four, two or one) x 32, 64 or 128 neighbouring queries share tiles of 64 keys, and two CTAs per SM hide each other's softmax.
//   warps 0-3  softmax, a thread per row: q to bf16 rows in shared memory once; per tile the scores from TMEM, capped / charged / masked as the
//              launch asks, fp32 maximum and sum; the weights go back to TMEM, over the scores and the columns behind them, as THREE bf16 terms
//              (24 bits; that body's two leave 2^-18). O stays in TMEM and is rescaled only when a row's maximum has grown by more than 2^8 since its last
//              reference. The tensor core truncates as it accumulates, so every kSaFlush tiles O is added, with ordinary rounding, to the row's place in
//              the scratch. Error of the result, that body | this one: 1.7e-6 | 8e-7 on prompts of up to 1000 tokens, 3.1e-6 | 1.5e-6 on one of 4096,
//              9.3e-6 | 2.7e-6 on 256 tokens behind 4000. (Two terms, nothing flushed: 1.84e-6, 3.3e-6, 9.4e-6 in 45, 372 and 258 us instead of 54, 468 and 339.)
//   warp 4     (one lane) TMA producer: boxes of 32 positions, looked up in the block table; boxes behind the portion's last position lie
//              outside the tensor map and read as zeros;
//   warp 5     (one lane) tcgen05.mma issuer: S = Q K^T, O += (hi + mid + lo) V with the weights read from TMEM, V MN-major as it lies;
//   warp 6     zeros the value rows between the last position and the end of its box (the pool may hold anything there).
// Bound: the fp32 work per score; the tensor pipe needs 1024 clocks per 128 x 64 scores at heads of 128. Caps and charges are applied in loops of
// their own: with tanhf and log1pf inlined 64 times the code left the instruction cache (210 us, then, where the loops took 81). Two scores per instruction where there is one
// that takes two, scores within a quarter of a cap through the series alone, the queries and the results moved in batches: prompts of 1000, 311, 700 and 37 tokens, 16 heads over 4
// of 128, capped at 30, 85 -> 63 us (launches one behind the other in a captured graph; capped at 2, where most tiles are beyond a quarter of it, 85 -> 81; not capped 57 -> 54).
// Clocks of a tile, capped: capping 1300, weights 1000, maximum 400, waiting for the products 2000; beside 4000 before the first
// and 6000 behind the last. Further figures: attention_run.
#include "seq_attn_decode.cuh"
#include "tcgen05.cuh"

namespace sllm {

constexpr int kSaRows = 128, kSaKeys = 64, kSaThreads = 256, kSaBox = 32;
constexpr int kSaFlush = 12;             // tiles between two flushes of O: from there on three terms' products would be further off than that body's two
constexpr uint32_t kSaTmem = 256;        // scores at 0 .. 63, then the weights' terms at 0 .. 95, O at 128; two CTAs share an SM's 512 columns
constexpr float kSaLog2e = 1.4426950408889634f;

// tanh to 1e-6 of its value without a branch: 1 - 2 / (1 + e^2|x|), and below 1/4, where that cancels, the Taylor series to x^9 (remainder 0.0089 x^11). The worst
// place is just above 1/4: the documented errors of ex2.approx (2^-22) and rcp.approx (1 ulp) and the rounding of 1 + e leave 2.2e-7 of a result of 0.245.
__device__ __forceinline__ float sa_tanh(float x) {
    const float a = fabsf(x), x2 = x * x;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + tc_exp2(a * (2.0f * kSaLog2e))));
    const float small = x * fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 62.0f / 2835.0f, -17.0f / 315.0f), 2.0f / 15.0f), -1.0f / 3.0f), 1.0f);
    return a < 0.25f ? small : copysignf(fmaf(-2.0f, r, 1.0f), x);
}
__device__ __forceinline__ float sa_log2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void sa_ld16(uint32_t taddr, uint32_t* o) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3]), "=r"(o[4]), "=r"(o[5]), "=r"(o[6]), "=r"(o[7]), "=r"(o[8]), "=r"(o[9]), "=r"(o[10]), "=r"(o[11]),
                   "=r"(o[12]), "=r"(o[13]), "=r"(o[14]), "=r"(o[15])
                 : "r"(taddr)
                 : "memory");
    tc_wait_ld();
#pragma unroll
    for (int e = 0; e < 16; ++e) asm volatile("" : "+r"(o[e]));
}

template <int HD>
struct SaShape {
    static constexpr int kBlocks = HD / 64, kQBlock = kSaRows * 128, kQBytes = kBlocks * kQBlock, kKBlock = kSaKeys * 128, kTile = kBlocks * kKBlock;
    static constexpr int kStages = HD == 128 ? 2 : 4;
    static constexpr int kSmem = 1024 + kQBytes + 2 * kStages * kTile + 512;
};

struct SaArgs {
    AttnArgs a;
    int hpc, hpc_log2, queries;          // query heads and queries of a CTA: hpc * queries = 128
    int vec_q;
    int32_t* status; unsigned polls;     // where a wait that was given up is reported, and after how many polls it is
};

template <int HD, bool kOpts>
__global__ void __launch_bounds__(kSaThreads, 2) seq_attention_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const SaArgs sa) {
    using Sh = SaShape<HD>;
    constexpr int ST = Sh::kStages;
    const AttnArgs& p = sa.a;
    const sllm_seq_batch& b = p.b;
    const int seg = b.qt_seg[blockIdx.x], off = b.qt_off[blockIdx.x], split = blockIdx.z;
    // The work list may hold any tiles of 32 queries. Those of one aligned run of `queries` that are in it are done together, by the CTA of the first of them:
    // bit i of `parts` says that the tile i behind this CTA's own is one of them.
    uint32_t parts = 1;
    const bool in_run = sa.queries > kBQ && off % kBQ == 0;
    if (in_run) {
        __shared__ uint32_t found;
        const int run = off & ~(sa.queries - 1);
        uint32_t mine = 0;
        for (int i = threadIdx.x; i < b.n_qtiles; i += kSaThreads) {
            const uint32_t d = (uint32_t)(b.qt_off[i] - run);
            if (b.qt_seg[i] == seg && d < (uint32_t)sa.queries && d % kBQ == 0) mine |= 1u << (d / kBQ);
        }
        if (threadIdx.x == 0) found = 0;
        __syncthreads();
        mine = __reduce_or_sync(0xffffffffu, mine);
        if (mine && threadIdx.x % 32 == 0) atomicOr(&found, mine);
        __syncthreads();
        const uint32_t own = 1u << ((off - run) / kBQ);
        if (found & (own - 1)) return;
        parts = found / own;
    }
    extern __shared__ uint8_t sa_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sa_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sK = smem, *sV = sK + ST * Sh::kTile, *sQ = sV + ST * Sh::kTile;
    uint64_t* kfull = reinterpret_cast<uint64_t*>(sQ + Sh::kQBytes);
    uint64_t *kempty = kfull + ST, *vfull = kempty + ST, *vready = vfull + ST, *vempty = vready + ST, *qready = vempty + ST, *sfull = qready + 1, *pready = sfull + 1, *odone = pready + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(odone + 1);
    volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = min((32 - __clz(parts)) * kBQ, b.seg_len[seg] - off), tok0 = b.seg_start[seg] + off, pos0 = b.seg_pos0[seg] + off, slot = b.seg_slot[seg];
    const int group = p.heads / p.kv_heads, sets = group / sa.hpc, gkv = blockIdx.y / sets, h0 = gkv * group + (blockIdx.y % sets) * sa.hpc;
    const int last_pos = pos0 + nq - 1;
    const TileList tiles(pos0, last_pos, seq_row_window(pos0, p.window, p.chunk), p.keep_first, kSaKeys);
    const int n = tiles.n > split ? (tiles.n - split + p.nsplit - 1) / p.nsplit : 0;      // this share's tiles: split, split + nsplit, ...

    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; ++i) { mb_init(kfull + i, 1); mb_init(kempty + i, 1); mb_init(vfull + i, 1); mb_init(vready + i, 1); mb_init(vempty + i, 1); }
        mb_init(qready, 128); mb_init(sfull, 1); mb_init(pready, 128); mb_init(odone, 1);
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tc_alloc(tmem_slot, kSaTmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int32_t* table = b.block_table + (size_t)slot * b.max_pages;

    if (warp == 4) {
        if (elect_one()) {   // ===== TMA producer =====
            for (int i = 0; i < n; ++i) {
                const int s = i % ST, j0 = tiles.tile_of(split + i * p.nsplit) * kSaKeys;
                const uint32_t ph = (uint32_t)(i / ST) & 1;
                int at[2], row[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int pos = j0 + x * kSaBox;
                    int in_page;
                    const int idx = page_of(pos, b.page_len, p.page_magic, in_page);
                    at[x] = pos <= last_pos ? in_page : b.page_len;                           // behind the last position: outside the map, zeros
                    row[x] = pos <= last_pos ? table[idx] * p.kv_heads + gkv : 0;
                }
                if (!tc_wait(kempty + s, ph ^ 1, gave_up, sa.polls)) break;
                mb_expect(kfull + s, Sh::kTile);
#pragma unroll
                for (int x = 0; x < 2; ++x)
                    for (int c = 0; c < Sh::kBlocks; ++c) tma_load_3d(sK + s * Sh::kTile + c * Sh::kKBlock + x * kSaBox * 128, &tmK, 64 * c, at[x], row[x], kfull + s);
                if (!tc_wait(vempty + s, ph ^ 1, gave_up, sa.polls)) break;
                mb_expect(vfull + s, Sh::kTile);
#pragma unroll
                for (int x = 0; x < 2; ++x)
                    for (int c = 0; c < Sh::kBlocks; ++c) tma_load_3d(sV + s * Sh::kTile + c * Sh::kKBlock + x * kSaBox * 128, &tmV, 64 * c, at[x], row[x], vfull + s);
            }
        }
    } else if (warp == 5) {
        if (elect_one()) {   // ===== MMA issuer: products of a tile leave one after the other only where their descriptors are at hand (made anew for each they took 60 clocks apiece, =====
                             // a tile's scores twice as long as the tensor pipe needs for them) =====
            constexpr uint32_t idesc_s = umma_idesc_bf16(kSaRows, kSaKeys), idesc_o = umma_idesc_bf16(kSaRows, HD) | (1u << 16);      // B MN-major
            const uint64_t q_desc = umma_desc_sw128(sQ), k_desc = umma_desc_sw128(sK), v_desc = umma_desc_mn_sw128(sV, Sh::kKBlock);  // + bytes / 16: another place
            auto scores = [&](int i) {
                const uint64_t k = k_desc + (uint32_t)(i % ST) * (Sh::kTile / 16);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks)
                    tc_mma_bf16(tmem, q_desc + (uint32_t)((ks / 4) * (Sh::kQBlock / 16) + 2 * (ks % 4)), k + (uint32_t)((ks / 4) * (Sh::kKBlock / 16) + 2 * (ks % 4)), idesc_s, ks != 0);
                tc_commit(sfull);
                tc_commit(kempty + i % ST);
            };
            bool ok = n > 0 && tc_wait(qready, 0, gave_up, sa.polls) && tc_wait(kfull, 0, gave_up, sa.polls);
            if (ok) {
                tc_fence_after();
                scores(0);
            }
            for (int i = 0; ok && i < n; ++i) {
                ok = tc_wait(vready + i % ST, (uint32_t)(i / ST) & 1, gave_up, sa.polls) && tc_wait(pready, (uint32_t)i & 1, gave_up, sa.polls);
                if (!ok) break;
                tc_fence_after();
                const uint64_t v = v_desc + (uint32_t)(i % ST) * (Sh::kTile / 16);
#pragma unroll
                for (int ks = 0; ks < 3 * kSaKeys / 16; ++ks)                    // first terms, then second ones, then third ones, against the same values
                    tc_mma_bf16_ts(tmem + 128, tmem + 8 * ks, v + (uint32_t)((ks % (kSaKeys / 16)) * 128), idesc_o, (i % kSaFlush | ks) != 0);
                tc_commit(odone);
                tc_commit(vempty + i % ST);
                if (i + 1 < n) {        // the next scores land where the weights lie that this product is still reading
                    ok = tc_wait(kfull + (i + 1) % ST, (uint32_t)((i + 1) / ST) & 1, gave_up, sa.polls) && tc_wait(odone, (uint32_t)i & 1, gave_up, sa.polls);
                    if (!ok) break;
                    tc_fence_after();
                    scores(i + 1);
                }
            }
        }
    } else if (warp == 6) {   // ===== value rows that the sequence does not have yet =====
        for (int i = 0; i < n; ++i) {
            const int s = i % ST, have = last_pos + 1 - tiles.tile_of(split + i * p.nsplit) * kSaKeys;
            if (!tc_wait_warp(vfull + s, (uint32_t)(i / ST) & 1, gave_up, sa.polls)) break;
            if (have < kSaKeys) {
                for (int x = lane; x < (kSaKeys - have) * 8 * Sh::kBlocks; x += 32) {
                    const int c = x / ((kSaKeys - have) * 8), y = x % ((kSaKeys - have) * 8);
                    *reinterpret_cast<uint4*>(sV + s * Sh::kTile + c * Sh::kKBlock + (have + y / 8) * 128 + (y % 8) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) mb_arrive(vready + s);
        }
    } else if (warp < 4) {   // ===== softmax: row = warp * 32 + lane = query * hpc + head =====
        const int row = threadIdx.x, qi = row >> sa.hpc_log2, h = h0 + (row & (sa.hpc - 1));
        const bool live = qi < nq && (parts >> (qi / kBQ) & 1);
        const int qpos = pos0 + qi;
        {   // the warp's 32 rows, one row (or two) per load so that neighbouring lanes read neighbouring columns
            constexpr int kLanes = HD / 4, kPer = 32 / kLanes;                  // lanes of a row, rows of a load
            // Sixteen loads on their way before the first of them is stored: left to itself the compiler keeps every load behind the store before it, since both could be
            // the same memory, and the queries of a CTA took 11000 to 21000 clocks.
            constexpr int kAhead = 16;
            const int col = (lane % kLanes) * 4;
#pragma unroll 1
            for (int r0 = 0; r0 < 32; r0 += kPer * kAhead) {
                float4 x[kAhead];
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    const int r = warp * 32 + r0 + k * kPer + lane / kLanes;
                    const float* src = p.q + (size_t)(tok0 + min(r >> sa.hpc_log2, nq - 1)) * p.ldq + (size_t)(h0 + (r & (sa.hpc - 1))) * HD + col;
                    if (sa.vec_q) x[k] = *reinterpret_cast<const float4*>(src);
                    else x[k] = make_float4(src[0], src[1], src[2], src[3]);
                }
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    const int r = warp * 32 + r0 + k * kPer + lane / kLanes;
                    *reinterpret_cast<uint2*>(sQ + (col / 64) * Sh::kQBlock + r * 128 + ((((col % 64) / 8) ^ (r & 7)) << 4) + (col % 8) * 2) =
                        make_uint2(tc_pack(x[k].x, x[k].y), tc_pack(x[k].z, x[k].w));
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mb_arrive(qready);
        }
        const uint32_t s_tmem = tmem + ((uint32_t)(warp * 32) << 16), o_tmem = s_tmem + 128;
        const int wnd = seq_row_window(qpos, p.window, p.chunk);
        const float slope = kOpts && p.slopes ? p.slopes[h] : 0.0f, r1 = kOpts && p.logdist ? p.logdist[h] : 0.0f, r2 = kOpts && p.logdist ? p.logdist[p.heads + h] : 0.0f;
        // Weights are 2^(score * mul - ref): one rounding between a score and its exponential. Without caps or charges mul holds the scale, too.
        const bool plain = !kOpts && p.scale > 0.0f;
        const float mul = plain ? p.scale * kSaLog2e : kSaLog2e;
        float ref = -INFINITY, l = 0.0f, flushed = -INFINITY;      // what the weights are relative to; their sum; the reference of what has been flushed
        const int rows = parts >> ((warp * 32 >> sa.hpc_log2) / kBQ) & 1 ? min(32, (nq << sa.hpc_log2) - warp * 32) : 0;      // a warp's rows belong to one tile
        // the records of this warp's rows, and how far the next head's and the next query's are
        float* recs = p.ws + (((size_t)tok0 * p.heads + h0) * p.nsplit + split) * (HD + 2);
        const int rec_h = p.nsplit * (HD + 2), rec_q = p.heads * rec_h;
        auto rec_of = [&](int r) { return recs + (size_t)(uint32_t)(((warp * 32 + r) >> sa.hpc_log2) * rec_q + ((warp * 32 + r) & (sa.hpc - 1)) * rec_h); };
        // Where this row's sums are flushed to, 16 columns at a time. Rows of its own when a record follows; when the result does, all the records of the query's heads are
        // free, and the heads' lanes take turns of 16 bytes there so that a store covers whole sectors.
        const bool direct = p.out || p.out16;
        const int turn = direct ? sa.hpc : 1, hh = row & (sa.hpc - 1);
        float* place = direct ? reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(rec_of(lane) - hh * rec_h) + 15) & ~(uintptr_t)15) + 4 * hh : rec_of(lane) + 2;
        auto prefetch_flushed = [&]() {
            const float* line = direct ? place - 4 * hh + hh * HD : place;
#pragma unroll
            for (int c = 0; c < HD; c += 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(line + c));
        };
        auto store_flushed = [&](const uint32_t* o, int c) {
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
                float* at = place + (c + e) * turn;
                if (direct) {
                    *reinterpret_cast<uint4*>(at) = make_uint4(o[e], o[e + 1], o[e + 2], o[e + 3]);
                } else {
                    *reinterpret_cast<uint2*>(at) = make_uint2(o[e], o[e + 1]);
                    *reinterpret_cast<uint2*>(at + 2) = make_uint2(o[e + 2], o[e + 3]);
                }
            }
        };
        auto add_flushed = [&](uint32_t* o, int c) {        // carried over to the present reference
            const float f = flushed == ref ? 1.0f : tc_exp2(flushed - ref);
            float4 w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* at = place + (c + 4 * e) * turn;
                if (direct) {
                    w[e] = *reinterpret_cast<const float4*>(at);
                } else {
                    const float2 a = *reinterpret_cast<const float2*>(at), b2 = *reinterpret_cast<const float2*>(at + 2);
                    w[e] = make_float4(a.x, a.y, b2.x, b2.y);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[4 * e] = __float_as_uint(fmaf(w[e].x, f, __uint_as_float(o[4 * e])));
                o[4 * e + 1] = __float_as_uint(fmaf(w[e].y, f, __uint_as_float(o[4 * e + 1])));
                o[4 * e + 2] = __float_as_uint(fmaf(w[e].z, f, __uint_as_float(o[4 * e + 2])));
                o[4 * e + 3] = __float_as_uint(fmaf(w[e].w, f, __uint_as_float(o[4 * e + 3])));
            }
        };
        bool ok = true;
        for (int i = 0; i < n; ++i) {
            const int j0 = tiles.tile_of(split + i * p.nsplit) * kSaKeys;
            ok = tc_wait_warp(sfull, (uint32_t)i & 1, gave_up, sa.polls);
            if (!ok) break;
            tc_fence_after();
            uint32_t s[64];
            tc_ld32_async(s_tmem, s);
            tc_ld32_async(s_tmem + 32, s + 32);
            tc_arrived(s);
            tc_arrived(s + 32);
            // every key of the tile is visible to every row of the warp
            const bool all = __all_sync(0xffffffffu, j0 + kSaKeys - 1 <= qpos && (qpos - j0 < wnd || j0 + kSaKeys <= p.keep_first));
            if (kOpts && p.softcap > 0.0f) {
                const float inv = p.scale / p.softcap;
                const uint64_t inv2 = tc_two(__float_as_uint(inv), __float_as_uint(inv));
                float top0 = 0.0f, top1 = 0.0f;
#pragma unroll
                for (int e = 0; e < 64; e += 2) {
                    float x, y;
                    tc_split(tc_mul2(tc_two(s[e], s[e + 1]), inv2), x, y);
                    s[e] = __float_as_uint(x);
                    s[e + 1] = __float_as_uint(y);
                    if (e & 2) top1 = tc_max3(top1, fabsf(x), fabsf(y));
                    else top0 = tc_max3(top0, fabsf(x), fabsf(y));
                }
                // Scores within a quarter of the cap, as nearly all are: the series alone, two at a time. It is the one sa_tanh takes for them, so which of the two loops a tile
                // goes through shows in no bit (NaN stays NaN in both).
                if (__any_sync(0xffffffffu, fmaxf(top0, top1) >= 0.25f)) {
#pragma unroll
                    for (int e = 0; e < 64; ++e) s[e] = __float_as_uint(p.softcap * sa_tanh(__uint_as_float(s[e])));
                } else {
                    auto both = [](float v) { return tc_two(__float_as_uint(v), __float_as_uint(v)); };
                    const uint64_t c4 = both(62.0f / 2835.0f), c3 = both(-17.0f / 315.0f), c2 = both(2.0f / 15.0f), c1 = both(-1.0f / 3.0f), c0 = both(1.0f), cap2 = both(p.softcap);
#pragma unroll
                    for (int e = 0; e < 64; e += 2) {
                        const uint64_t x = tc_two(s[e], s[e + 1]), x2 = tc_mul2(x, x);
                        float a, c;
                        tc_split(tc_mul2(cap2, tc_mul2(x, tc_fma2(x2, tc_fma2(x2, tc_fma2(x2, tc_fma2(x2, c4, c3), c2), c1), c0))), a, c);
                        s[e] = __float_as_uint(a);
                        s[e + 1] = __float_as_uint(c);
                    }
                }
            } else if (!plain) {
#pragma unroll
                for (int e = 0; e < 64; ++e) s[e] = __float_as_uint(__uint_as_float(s[e]) * p.scale);
            }
            if (kOpts && p.slopes) {
                const float d0 = (float)(qpos - j0);
#pragma unroll
                for (int e = 0; e < 64; ++e) s[e] = __float_as_uint(fmaf(-slope, d0 - (float)e, __uint_as_float(s[e])));
            }
            if (kOpts && p.logdist) {
                const float d0 = (float)(qpos - j0), r1l = r1 * 0.6931471805599453f;
#pragma unroll
                for (int e = 0; e < 64; ++e) s[e] = __float_as_uint(fmaf(-r1l, sa_log2(fmaf(r2, fmaxf(d0 - (float)e, 0.0f), 1.0f)), __uint_as_float(s[e])));
            }
            if (!all) {
#pragma unroll
                for (int e = 0; e < 64; ++e)
                    if (!seq_sees(qpos, j0 + e, wnd, p.keep_first)) s[e] = 0xff800000u;       // -inf
            }
            float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < 64; e += 2) m[(e / 2) & 3] = tc_max3(m[(e / 2) & 3], __uint_as_float(s[e]), __uint_as_float(s[e + 1]));
            const float mx = tc_max3(fmaxf(m[0], m[1]), m[2], m[3]) * mul;
            if (i % kSaFlush == 0 && i > 0) {           // the product before this tile has completed: these scores follow it
                if (live && i > kSaFlush) prefetch_flushed();
#pragma unroll 1
                for (int c = 0; c < HD; c += 16) {
                    uint32_t o[16];
                    sa_ld16(o_tmem + c, o);
                    if (live) {
                        if (i > kSaFlush) add_flushed(o, c);
                        store_flushed(o, c);
                    }
                    __syncwarp();
                }
                flushed = ref;
            }
            if (i == 0) {
                ref = mx;
            } else if (__any_sync(0xffffffffu, mx > ref + 8.0f)) {
                const float nr = fmaxf(ref, mx), f = nr == ref ? 1.0f : tc_exp2(ref - nr);
                l *= f;
                ref = nr;
#pragma unroll 1
                for (int c = 0; c < HD; c += 16) {
                    uint32_t o[16];
                    sa_ld16(o_tmem + c, o);
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                    tc_st16(o_tmem + c, o);
                }
            }
            uint64_t sum = 0;                                                   // (0, 0)
            const float from = ref == -INFINITY ? 0.0f : ref;                   // nothing seen yet: every weight is exp(-inf) = 0
            const uint64_t mul2 = tc_two(__float_as_uint(mul), __float_as_uint(mul)), from2 = tc_two(__float_as_uint(-from), __float_as_uint(-from));
            const uint64_t less = tc_two(__float_as_uint(-1.0f), __float_as_uint(-1.0f));
            auto terms = [](uint32_t w) { return tc_two(w << 16, w & 0xffff0000u); };
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t hi[16], mid[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float x, y;
                    tc_split(tc_fma2(tc_two(s[half * 32 + 2 * e], s[half * 32 + 2 * e + 1]), mul2, from2), x, y);
                    x = tc_exp2(x);
                    y = tc_exp2(y);
                    const uint64_t w = tc_two(__float_as_uint(x), __float_as_uint(y));
                    sum = tc_add2(sum, w);
                    hi[e] = tc_pack(x, y);
                    const uint64_t r = tc_fma2(terms(hi[e]), less, w);          // what the first terms leave: exact
                    tc_split(r, x, y);
                    mid[e] = tc_pack(x, y);
                    tc_split(tc_fma2(terms(mid[e]), less, r), x, y);
                    lo[e] = tc_pack(x, y);
                }
                tc_st16(s_tmem + half * 16, hi);
                tc_st16(s_tmem + 32 + half * 16, mid);
                tc_st16(s_tmem + 64 + half * 16, lo);
            }
            float l0, l1;
            tc_split(sum, l0, l1);
            l += l0 + l1;
            tc_wait_st();
            tc_fence_before();
            mb_arrive(pready);
        }
        if (live && n > kSaFlush) prefetch_flushed();
        if (ok && n > 0) ok = tc_wait_warp(odone, (uint32_t)(n - 1) & 1, gave_up, sa.polls);
        tc_fence_after();
        float inv = direct ? 1.0f / l : 1.0f;
        const int t = tok0 + qi;
        if (ok && live && !direct) {
            // the reference as a logarithm to the base e, and what its rounding leaves of it in the sums
            constexpr float ln2 = 0.693147181f, ln2_rest = -1.90465421e-9f;
            const float m = ref * ln2;
            if (ref != -INFINITY) inv = 1.0f + fmaf(ref, ln2_rest, fmaf(ref, ln2, -m));
            rec_of(lane)[0] = m;
            rec_of(lane)[1] = l * inv;
        }
        float* mine = reinterpret_cast<float*>(smem) + warp * (32 * 33);        // the rings' place: every tile has been read
        // fp32 results: where this lane's column of the first row goes, and how far the next query and the next head are
        float* to = lane + (p.out ? p.out + (size_t)tok0 * p.ldo + (size_t)h0 * HD : recs + 2);
        const int step_h = p.out ? HD : rec_h, step_q = p.out ? p.ldo : rec_q;
#pragma unroll 1
        for (int c = 0; ok && c < HD; c += 32) {
            uint32_t o[32];
            if (n > 0) {
                tc_ld32_async(o_tmem + c, o);
                tc_arrived(o);
            } else {
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] = 0u;
            }
            if (n > kSaFlush && live) {
                add_flushed(o, c);
                add_flushed(o + 16, c + 16);
            }
            __syncwarp();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * inv);
            if (live && p.out16) {
                uint4* dst = reinterpret_cast<uint4*>(p.out16 + ((size_t)t * p.heads + h) * HD + c);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    auto two = [&](int e) { return tc_pack(__uint_as_float(o[8 * x + e]), __uint_as_float(o[8 * x + e + 1])); };
                    dst[x] = make_uint4(two(0), two(2), two(4), two(6));
                }
            }
            if (p.out || !direct) {     // fp32 rows: through shared memory, so that a store covers neighbouring columns of one row
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 32; ++e) mine[lane * 33 + e] = __uint_as_float(o[e]);
                __syncwarp();
#pragma unroll 1
                for (int r0 = 0; r0 < rows; r0 += 16) {                        // sixteen rows read before the first is stored, as above
                    float x[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) x[k] = mine[(r0 + k) * 33 + lane];
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const int rr = warp * 32 + r0 + k;
                        if (r0 + k < rows) to[(size_t)(uint32_t)((rr >> sa.hpc_log2) * step_q + (rr & (sa.hpc - 1)) * step_h + c)] = x[k];
                    }
                }
            }
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*gave_up) tc_gave_up(sa.status);
    if (warp == 5) {
        tc_fence_after();
        tc_dealloc(tmem, kSaTmem);
    }
}

template <int HD, bool kOpts>
static int sa_launch(const AttnArgs& p, cudaStream_t st) {
    using Sh = SaShape<HD>;
    auto* kernel = seq_attention_tc_kernel<HD, kOpts>;
    static bool configured = false;
    if (!configured) {
        SLLM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
        configured = true;
    }
    SaArgs a{};
    a.a = p;
    const int group = p.heads / p.kv_heads;
    a.hpc = group % 4 == 0 ? 4 : group % 2 == 0 ? 2 : 1;
    a.hpc_log2 = a.hpc / 2;
    a.queries = kSaRows / a.hpc;
    if (int rc = status_check()) return rc;
    if (int rc = status_word(&a.status)) return rc;
    a.polls = (unsigned)g_tune_tc_polls;
    a.vec_q = p.ldq % 4 == 0 && ((uintptr_t)p.q % 16) == 0;
    // a pool [pages][kv_heads][page_len][HD]: how many pages it has is the caller's knowledge, the block table names existing ones only
    CUtensorMap tmK, tmV;
    const cuuint64_t dims[3] = {HD, (cuuint64_t)p.b.page_len, (cuuint64_t)1 << 31};
    const cuuint64_t strides[2] = {HD * 2, (cuuint64_t)p.b.page_len * HD * 2};
    const cuuint32_t box[3] = {64, kSaBox, 1};
    if (int rc = tc_encode_bf16(&tmK, p.k_pool, 3, dims, strides, box)) return rc;
    if (int rc = tc_encode_bf16(&tmV, p.v_pool, 3, dims, strides, box)) return rc;
    kernel<<<dim3(p.b.n_qtiles, p.heads / a.hpc, p.nsplit), kSaThreads, Sh::kSmem, st>>>(tmK, tmV, a);
    ++g_launches;
    SLLM_LAUNCH_CHECK_ONLY();
    return SLLM_OK;
}

int launch_attention_tc(const AttnArgs& p, cudaStream_t st) {
    const bool opts = p.softcap > 0.0f || p.slopes || p.logdist;
    if (p.dk == 128) return opts ? sa_launch<128, true>(p, st) : sa_launch<128, false>(p, st);
    return opts ? sa_launch<64, true>(p, st) : sa_launch<64, false>(p, st);
}

}  // namespace sllm
