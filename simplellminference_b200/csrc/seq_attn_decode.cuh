// csrc/seq_attn_decode.cuh — attention of steps of single tokens (decoding) over the paged cache; part of seq_attn.cu.
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "seq_attn.cuh"

namespace sllm {

struct AttnArgs {
    sllm_seq_batch b;
    const float* q; int ldq, heads, kv_heads, dk, dv; float scale;
    const void *k_pool, *v_pool;
    int nsplit; float* ws;
    int by_head;   // fp32 body, steps of single tokens: a CTA's "queries" are the query heads of ONE kv head at one token (they share its tiles)
    int window, keep_first;   // query i sees key j <= i when i - j < window or j < keep_first (window INT_MAX = everything before it)
    float softcap;            // > 0: score <- softcap * tanh(score / softcap)
    const float* slopes;      // [heads] or NULL: score <- score - slopes[h] * (i - j)
    int v_in_k;               // values = the first dv columns of the key rows (v_pool unused)
    const float* logdist;     // [2][heads] or NULL: score <- score - r1[h] * ln(1 + r2[h] * (i - j)), r1 = row 0, r2 = row 1
    // Every query head's weights on every key/value head's values: `heads` then counts kv_heads * q_heads results, result u = (value
    // head u / q_heads, query head u % q_heads); the query head reads the KEYS of its own key/value head as always. Otherwise q_heads = heads.
    int q_heads, cross;
    int chunk;                // > 0: a query sees its own chunk of `chunk` positions only (then window / keep_first are not used)
    float* out; int ldo; uint16_t* out16;   // one share: the normalised result goes here (fp32 [T][ldo] and / or dense bf16) instead of ws
    uint32_t page_magic;      // ceil(2^32 / page_len): the page of a position without a division (page_of)
    int by_request;           // decode over bf16 pools: the grid has the requests in x (more of them than y takes)
};

// prompt portions over bf16 pools on tcgen05: dk = dv = 64 or 128, pools 16-byte aligned, no values inside keys, no cross values (seq_attn_tc.cu)
int launch_attention_tc(const AttnArgs& p, cudaStream_t st);

#ifdef __CUDACC__

__device__ __forceinline__ float seq_score(float dot, float scale, float softcap, float slope, float r1, float r2, int qpos, int key) {
    float sc = dot * scale;
    if (softcap > 0.0f) sc = softcap * tanhf(sc / softcap);
    sc -= slope * (float)(qpos - key);
    if (r1 != 0.0f) sc -= r1 * log1pf(r2 * (float)(qpos - key));
    return sc;
}

// page of a position and its row there: the product with the rounded-up reciprocal is at most one too large
__device__ __forceinline__ int page_of(int pos, int page_len, uint32_t magic, int& in_page) {
    int page = (int)__umulhi((uint32_t)pos, magic);
    in_page = pos - page * page_len;
    if (in_page < 0) {
        --page;
        in_page += page_len;
    }
    return page;
}

// 16 bytes of a cache row as pairs of floats
__device__ __forceinline__ void cache_pairs(const uint4& u, uint64_t (&p)[2]) {
    p[0] = pair_f32(u.x, u.y);
    p[1] = pair_f32(u.z, u.w);
}

constexpr int kDecodeWarps = 4, kDecodeCluster = 16;     // warps of a CTA, CTAs of a cluster at most

// fp32 pools. One query per sequence: G query heads of one kv head against that head's cache rows. Bound: HBM (each row is read once and used G times), so
// rows go from global memory to registers and nothing is staged: eight lanes share a row (16-byte loads, neighbours next to each other), the four
// groups of lanes of a warp hold neighbouring rows, kSteps of them in flight per lane, values requested before the scores are worked on. Everything
// is fp32 (queries as they are, two products per instruction); G x kSteps scores cross the eight lanes in one halving exchange, which leaves
// every score on one lane for its exponential. A sequence's rows are dealt in runs of 4 x kSteps keys to all warps of a thread-block cluster, so that
// the longest context of a step is spread over up to 16 CTAs whatever the step's share count; every warp sends its sums to the CTAs that own the
// columns (distributed shared memory, one barrier), which merge them and write the result (or one record per share when something still follows).
template <int L, int G, int kSteps>     // 16-byte loads per lane of a key or value row: heads of D = 32 L
__global__ void __launch_bounds__(kDecodeWarps * 32) seq_attention_decode_kernel(AttnArgs p) {
    after_previous();
    namespace cg = cooperative_groups;
    constexpr int E = 4, PE = E / 2, D = 8 * L * E, VAL = G * kSteps;
    constexpr int kPer = VAL >= 8 ? VAL / 8 : 1, kDup = VAL >= 8 ? 1 : 8 / VAL;      // scores per lane after the exchange, lanes that hold the same one
    constexpr int kRun = 4 * kSteps;                                                  // keys of one step of a warp
    static_assert(kBK % kRun == 0, "a run of keys lies inside one tile");
    constexpr int kPairs = G * L * PE;                  // pairs of sums a lane keeps
    // what the cluster's warps send this CTA: their sums for its share of the G * D results, and every warp's (maximum, sum) per head
    __shared__ __align__(16) float got_o[kDecodeWarps * G * D];
    __shared__ __align__(16) float2 got_ml[kDecodeCluster * kDecodeWarps][G];
    __shared__ float weight[kDecodeCluster * kDecodeWarps][G], total[G][2];
    const sllm_seq_batch& b = p.b;
    cg::cluster_group cluster = cg::this_cluster();
    const int CS = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), split = blockIdx.z / CS;
    cluster.barrier_arrive();       // waited for before anything is sent: every CTA of the cluster runs by then
    const int seg = b.qt_seg[blockIdx.x], t = b.seg_start[seg], pos = b.seg_pos0[seg], slot = b.seg_slot[seg];
    const int group = p.heads / p.kv_heads, subsets = group / G, gkv = blockIdx.y / subsets, h0 = gkv * group + (blockIdx.y % subsets) * G;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, j8 = lane & 7, kg = lane >> 3;
    const int wnd = seq_row_window(pos, p.window, p.chunk);
    const TileList tiles(pos, pos, wnd, p.keep_first, kBK);
    constexpr int kRuns = kBK / kRun;
    const int n_runs = tiles.n * kRuns, workers = p.nsplit * CS * kDecodeWarps;
    const float* kp = reinterpret_cast<const float*>(p.k_pool);
    const float* vp = reinterpret_cast<const float*>(p.v_pool);
    const int32_t* table = b.block_table + (size_t)slot * b.max_pages;

    uint64_t qv[G][L * PE];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < L; ++i) {
            const float* src = p.q + (size_t)t * p.ldq + (size_t)(h0 + g) * D + (i * 8 + j8) * E;
#pragma unroll
            for (int e = 0; e < PE; ++e) qv[g][i * PE + e] = pair_f32(src[2 * e], src[2 * e + 1]);
        }
    // this lane's scores: head og, steps os .. os + kPer - 1 of its group's keys
    const int og = (j8 / kDup) * kPer / kSteps, os = (j8 / kDup) * kPer % kSteps;
    const float slope = p.slopes ? p.slopes[h0 + og] : 0.0f;
    const float r1 = p.logdist ? p.logdist[h0 + og] : 0.0f, r2 = p.logdist ? p.logdist[p.heads + h0 + og] : 0.0f;
    float m[G], l = 0.0f;                       // running maxima (all lanes alike); this lane's share of the sum of head og
    uint64_t acc[G][L * PE];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY;
#pragma unroll
        for (int i = 0; i < L * PE; ++i) acc[g][i] = 0ull;
    }
    auto first_key = [&](int run) { return tiles.tile_of(run / kRuns) * kBK + run % kRuns * kRun; };
    // rows the sequence does not have yet read as zeros (their memory may hold anything)
    auto load_keys = [&](uint4 (&u)[kSteps][L], int j0, int page) {
        const float* row = kp + seq_pool_row(page, p.kv_heads, gkv, b.page_len, j0 % b.page_len + kg, D) + j8 * E;
#pragma unroll
        for (int s = 0; s < kSteps; ++s)
#pragma unroll
            for (int i = 0; i < L; ++i) u[s][i] = j0 + 4 * s + kg <= pos ? ld_stream(row + (size_t)(4 * s) * D + i * 8 * E) : make_uint4(0u, 0u, 0u, 0u);
    };
    auto load_values = [&](uint4 (&u)[kSteps][L], int j0, int page) {
        const float* row = vp + seq_pool_row(page, p.kv_heads, gkv, b.page_len, j0 % b.page_len + kg, D) + j8 * E;
#pragma unroll
        for (int s = 0; s < kSteps; ++s)
#pragma unroll
            for (int i = 0; i < L; ++i) u[s][i] = j0 + 4 * s + kg <= pos ? ld_stream(row + (size_t)(4 * s) * D + i * 8 * E) : make_uint4(0u, 0u, 0u, 0u);
    };
    // A run's keys are asked for as soon as the previous run's have been multiplied, its values likewise: one of the two is always on its way.
    uint4 ku[kSteps][L], vu[kSteps][L];
    int run = (split * CS + rank) * kDecodeWarps + warp, page = 0;
    if (run < n_runs) {
        const int j0 = first_key(run);
        const int first = table[j0 / b.page_len];
        if (run + workers < n_runs) page = table[first_key(run + workers) / b.page_len];
        load_keys(ku, j0, first);
        load_values(vu, j0, first);
    }
    while (run < n_runs) {
        const int j0 = first_key(run), next = run + workers, jn = next < n_runs ? first_key(next) : 0, page_n = page;
        if (next + workers < n_runs) page = table[first_key(next + workers) / b.page_len];
        float sc[VAL];
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            uint64_t d[G];
#pragma unroll
            for (int g = 0; g < G; ++g) d[g] = 0ull;
#pragma unroll
            for (int i = 0; i < L; ++i) {
                uint64_t kk[PE];
                cache_pairs(ku[s][i], kk);
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < PE; ++e) fma_pair(d[g], kk[e], qv[g][i * PE + e]);
            }
#pragma unroll
            for (int g = 0; g < G; ++g) sc[g * kSteps + s] = pair_sum(d[g]);
        }
        if (next < n_runs) load_keys(ku, jn, page_n);
#pragma unroll
        for (int n = VAL / 2, bit = 4; n >= kPer && bit >= kDup; n /= 2, bit /= 2) {
            const bool up = lane & bit;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float give = up ? sc[i] : sc[i + n], keep = up ? sc[i + n] : sc[i];
                sc[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
            }
        }
#pragma unroll
        for (int o = kDup / 2; o >= 1; o /= 2) sc[0] += __shfl_xor_sync(0xffffffffu, sc[0], o);
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int key = j0 + 4 * (os + i) + kg;
            sc[i] = seq_sees(pos, key, wnd, p.keep_first) ? seq_score(sc[i], p.scale, p.softcap, slope, r1, r2, pos, key) : -INFINITY;
            mx = fmaxf(mx, sc[i]);
        }
#pragma unroll
        for (int o = 1; o < 8 / G; o *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        float mn[G], mine = 0.0f, before = 0.0f;
        bool moved = false;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            mn[g] = fmaxf(m[g], __shfl_sync(0xffffffffu, mx, g * (8 / G)));
            moved |= mn[g] != m[g];
            if (g == og) { mine = mn[g]; before = m[g]; }
        }
        if (moved) {                            // the same answer on all lanes
            l *= mine == -INFINITY ? 1.0f : expf(before - mine);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float corr = mn[g] == -INFINITY ? 1.0f : expf(m[g] - mn[g]);
                const uint64_t c2 = pair_f32(corr, corr);
#pragma unroll
                for (int i = 0; i < L * PE; ++i) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[g][i]) : "l"(c2));
                m[g] = mn[g];
            }
        }
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            sc[i] = sc[i] == -INFINITY ? 0.0f : expf(sc[i] - mine);
            if (j8 % kDup == 0) l += sc[i];
        }
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            uint64_t w2[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int v = g * kSteps + s;
                const float w = __shfl_sync(0xffffffffu, sc[v % kPer], (lane & 24) + v / kPer * kDup);
                w2[g] = pair_f32(w, w);
            }
#pragma unroll
            for (int i = 0; i < L; ++i) {
                uint64_t vv[PE];
                cache_pairs(vu[s][i], vv);
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < PE; ++e) fma_pair(acc[g][i * PE + e], vv[e], w2[g]);
            }
        }
        if (next < n_runs) load_values(vu, jn, page_n);
        run = next;
    }
    // The warp's four groups of keys: in two exchanges a lane gives away three quarters of its pairs and gets the others' parts of the rest.
    uint64_t v[kPairs];
#pragma unroll
    for (int i = 0; i < kPairs; ++i) v[i] = acc[i / (L * PE)][i % (L * PE)];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int bit = half ? 8 : 16, n = half ? kPairs / 4 : kPairs / 2;
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < kPairs / 2; ++i)
            if (i < n) {
                const uint64_t give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i], other = __shfl_xor_sync(0xffffffffu, (unsigned long long)give, bit);
                asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v[i]) : "l"(keep), "l"(other));
            }
    }
    float lg[G];
#pragma unroll
    for (int g = 0; g < G; ++g) lg[g] = warp_sum(og == g ? l : 0.0f);
    // every CTA of the cluster gets the sums of its own share of the results, and everybody's maxima
    const int share = G * D / CS, worker = rank * kDecodeWarps + warp;
    cluster.barrier_wait();
#pragma unroll
    for (int i = 0; i < kPairs / 4; ++i) {
        const int at = kg * (kPairs / 4) + i, g = at / (L * PE), r = at % (L * PE);
        const int item = g * D + (r / PE * 8 + j8) * E + r % PE * 2, to = item / share;
        *reinterpret_cast<uint64_t*>(cluster.map_shared_rank(got_o, to) + worker * share + item % share) = v[i];
    }
    if (lane < CS) {
        float2* ml = cluster.map_shared_rank(&got_ml[0][0], lane) + worker * G;
#pragma unroll
        for (int g = 0; g < G; ++g) ml[g] = make_float2(m[g], lg[g]);
    }
    cluster.sync();
    if (warp < G) {
        const int n = CS * kDecodeWarps;
        float M = -INFINITY, sum = 0.0f;
        for (int i = lane; i < n; i += 32) M = fmaxf(M, got_ml[i][warp].x);
        M = warp_max(M);
        for (int i = lane; i < n; i += 32) {
            const float f = got_ml[i][warp].x == -INFINITY ? 0.0f : expf(got_ml[i][warp].x - M);
            weight[i][warp] = f;
            sum = fmaf(got_ml[i][warp].y, f, sum);
        }
        sum = warp_sum(sum);
        if (lane == 0) {
            total[warp][0] = M;
            total[warp][1] = sum;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < share; i += kDecodeWarps * 32) {
        const int item = rank * share + i, g = item / D, c = item % D;
        float o = 0.0f;
#pragma unroll 4
        for (int w = 0; w < CS * kDecodeWarps; ++w) o = fmaf(got_o[w * share + i], weight[w][g], o);
        if (p.out || p.out16) {
            o *= 1.0f / total[g][1];
            if (p.out) p.out[(size_t)t * p.ldo + (size_t)(h0 + g) * D + c] = o;
            if (p.out16) p.out16[((size_t)t * p.heads + h0 + g) * D + c] = f32_to_bf16_bits(o);
        } else {
            float* rec = p.ws + (((size_t)t * p.heads + h0 + g) * p.nsplit + split) * (D + 2);
            rec[2 + c] = o;
            if (c == 0) {
                rec[0] = total[g][0];
                rec[1] = total[g][1];
            }
        }
    }
}

// The same step over bf16 pools, on the tensor cores without giving up fp32 working accuracy. The body above spends 1100 instructions per 16 bf16 rows
// and four query heads (28 % of the issue slots busy with the two warps per scheduler its registers allow: 57 us on eight requests of 77 to
// 8000 positions); mma.sync does the same in some 460 with the softmax and the loads (40 us; 32 requests of 2048 positions 84 -> 47 us, 5.7 TB/s). Operands: cache rows are bf16 as they are; every query value is the sum of three bf16 terms (24 bits), and
// the three terms of up to four heads are the 16 rows of the A fragment (row 2h first term, 2h + 1 second, 8 + 2h third), so S costs no more
// products than one bf16 query would; the softmax weights are split the same way and land in the A fragment of the second product without
// leaving their lane. Sums: products of bf16 terms are exact, a chain is at most two instructions long (32 products) before it is added to an fp32
// register with ordinary rounding, because the tensor core's own accumulation truncates. Rows come in runs of 16 through a ring of kRing stages per
// warp (cp.async, chunks swizzled for ldmatrix), no barrier between warps until the merge, which is that of the register body.
template <int D>
struct DecodeTile {
    static constexpr int kRun = 16, kRing = D == 128 ? 3 : 6;                    // keys of a stage, stages (two CTAs per SM)
    static constexpr int kStage = 2 * kRun * D;                                 // key rows, then value rows; 16-byte chunk i of row r lies at i ^ (r % 8)
    static constexpr int kSmem = kDecodeWarps * kRing * kStage * 2;
};

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// What a second turn of a cluster costs, in runs of 16 keys a warp
constexpr float kTurnRuns = 4.0f;

// kOpts: capped scores or charges on the distance (a window, kept positions and chunks are part of both). kPair: 0 = a cluster has one item (a request and a set of heads), the grid is
// (sets, requests) or, with by_request, (requests, sets); else it has those of two requests, the x-th and the x-th from the back of the caller's list (the longest context first), and
// kPair = 2: it has two CTAs.
// A step's clusters are all resident at once. With one item each, requests of unequal length leave most of the machine idle behind the longest; a pair divides its CTAs by what the two
// contexts need and, where that leaves the longer one too few, takes them one behind the other with all of them. Clusters look at their own pair only. Measured, us in a captured graph, one item a
// cluster | pairs, contexts of 16 to 8000 positions, 32 heads over 8 of 128: five requests 28.4 | 23.1, eight 36.1 | 27.4, 13 57.9 | 35.7, 32 95.5 | 61.9; requests alike, whose pairs only cost (barriers of larger
// clusters): eight of 64, 1000 and 2048 7.0 | 7.0, 11.7 | 11.9, 18.0 | 18.1, 16 of 300 9.4 | 9.9, 13 of 6000 59.9 | 62.9; 8 heads over 8 of 64: eight of 64 and 1000 5.5 | 5.7, 8.2 | 8.5, 13 of 300 7.0 | 7.5, 32 of 64
// 5.5 | 5.7. (Twice as many clusters as fit at once, half of which left again where requests are alike: 21.9, 25.6, 36.6, 58.5; alike 8.9, 13.2, 19.3, 11.3, 72.4; 7.4, 10.3, 8.4, 7.7.)
template <int D, bool kOpts, int kPair>
__global__ void __launch_bounds__(kDecodeWarps * 32, 2) seq_attention_decode_mma_kernel(AttnArgs p, int G) {
    static_assert(kDecodeWarps == 4, "sums of a column");
    after_previous();
    namespace cg = cooperative_groups;
    using Tile = DecodeTile<D>;
    constexpr int kRun = Tile::kRun, kRing = Tile::kRing, kSteps = D / 16, kTiles = D / 8;
    extern __shared__ __align__(16) uint16_t dsm[];
    __shared__ __align__(16) float got_o[kDecodeWarps * (4 * D + (kPair ? 16 : 0))];      // (a cluster's share of an item may be any number of CTAs up to eight)
    __shared__ __align__(16) float2 got_ml[kDecodeCluster * kDecodeWarps * 4];
    __shared__ float weight[kDecodeCluster * kDecodeWarps][4], total[4][2];
    const sllm_seq_batch& b = p.b;
    cg::cluster_group cluster = cg::this_cluster();
    const int full = (int)cluster.num_blocks(), split = blockIdx.z / full;
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // waited for before anything is sent: every CTA of the cluster runs by then (nothing is handed over)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3, h = g >> 1;
    struct Item { int t, pos, slot; };
    auto look_up = [&](int x) {
        const int seg = b.qt_seg[x];
        return Item{b.seg_start[seg], b.seg_pos0[seg], b.seg_slot[seg]};
    };
    auto runs_of = [&](int pos) { return TileList(pos, pos, seq_row_window(pos, p.window, p.chunk), p.keep_first, kBK).n * (kBK / kRun); };
    const bool swapped = !kPair && p.by_request;
    Item item = look_up(swapped ? blockIdx.x : blockIdx.y), next{};
    const int set = swapped ? blockIdx.y : blockIdx.x;
    int CS = full, base_rank = 0, turns = 1;
    if constexpr (kPair != 0) {
        const int other = b.n_qtiles - 1 - (int)blockIdx.y;
        next = look_up(other);
        if (other != (int)blockIdx.y) {
            const int a = runs_of(item.pos), z = runs_of(next.pos);
            int first = full / 2;      // CTAs of the first item: as many as end it with the other, one at least for either
            if (a != z) {
                first = min(full - 1, max(1, (int)((float)(a * full) / (float)(a + z) + 0.5f)));
                const float apart = fmaxf((float)a / (float)first, (float)z / (float)(full - first));
                if (apart * (float)full - (float)(a + z) > kTurnRuns * (float)(full * kDecodeWarps * p.nsplit)) turns = 2;
            }
            if (turns == 1) {
                const bool mine = (int)cluster.block_rank() < first;
                CS = mine ? first : full - first;
                base_rank = mine ? 0 : first;
                if (!mine) item = next;
            }
        }
    }
    const bool alone = kPair == 2 && CS == 1;       // nobody in the cluster waits for anybody
    const int rank = (int)cluster.block_rank() - base_rank;
    const int group = p.heads / p.kv_heads, subsets = group / G, gkv = set / subsets, h0 = gkv * group + (set % subsets) * G;
    const bool live = h < G, second = g & 1;           // this lane's head exists; it holds the second terms (and no third ones)
#pragma unroll 1
    for (int turn = 0; turn < (kPair ? turns : 1); ++turn) {
    if (turn) {
        cluster.barrier_arrive();   // what was sent to this thread in the turn before has been read
        item = next;
    }
    const int t = item.t, pos = item.pos, slot = item.slot;
    const int wnd = seq_row_window(pos, p.window, p.chunk);
    const TileList tiles(pos, pos, wnd, p.keep_first, kBK);
    const int n_runs = tiles.n * (kBK / kRun), workers = p.nsplit * CS * kDecodeWarps;
    const int32_t* table = b.block_table + (size_t)slot * b.max_pages;
    const uint16_t* kp = reinterpret_cast<const uint16_t*>(p.k_pool);
    const uint16_t* vp = reinterpret_cast<const uint16_t*>(p.v_pool);
    auto first_key = [&](int run) { return tiles.tile_of(run / (kBK / kRun)) * kBK + run % (kBK / kRun) * kRun; };

    // run -> stage of this warp's ring; rows the sequence does not have yet become zeros (their memory may hold anything)
    const uint32_t ring = smem_u32(dsm) + warp * (kRing * Tile::kStage * 2);
    constexpr int kChunks = D / 8, kPer = 32 / kChunks;          // 16-byte chunks of a row, rows one instruction of the warp brings
    const int lr = lane / kChunks, lc = lane % kChunks;
    const uint16_t* kl = kp + lc * 8;
    const uint16_t* vl = vp + lc * 8;
    auto issue = [&](int run, int stage) {
        if (run < n_runs) {
            const int j0 = first_key(run);
            int in_page;
            const int page = table[page_of(j0, b.page_len, p.page_magic, in_page)];
            const size_t row = seq_pool_row(page, p.kv_heads, gkv, b.page_len, in_page + lr, D);
            const uint16_t *ks = kl + row, *vs = vl + row;
            const uint32_t dst = ring + (stage * Tile::kStage + lr * D) * 2;
            const int have = pos - j0 - lr;           // row i * kPer of this lane exists when that is at least i * kPer
#pragma unroll
            for (int i = 0; i < kRun / kPer; ++i) {
                const uint32_t at = dst + i * kPer * D * 2 + ((lc ^ ((lr + i * kPer) & 7)) << 4);
                const int bytes = have >= i * kPer ? 16 : 0;         // (the rows of a run lie in one page: the address is good either way)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(ks + i * kPer * D), "r"(bytes) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + kRun * D * 2), "l"(vs + i * kPer * D), "r"(bytes) : "memory");
            }
        }
        cp_async_commit();
    };
    const int first_run = (split * CS + rank) * kDecodeWarps + warp;
#pragma unroll
    for (int i = 0; i < kRing - 1; ++i) issue(first_run + i * workers, i);

    uint32_t qa[kSteps][4];
    {
        const float* src = p.q + (size_t)t * p.ldq + (size_t)(h0 + (live ? h : 0)) * D + 2 * c;
#pragma unroll
        for (int ks = 0; ks < kSteps; ++ks)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t t1, t2, t3;
                split3_bf16(src[ks * 16 + half * 8], src[ks * 16 + half * 8 + 1], t1, t2, t3);
                qa[ks][half * 2] = !live ? 0u : second ? t2 : t1;
                qa[ks][half * 2 + 1] = !live || second ? 0u : t3;
            }
    }
    const float slope = p.slopes && live ? p.slopes[h0 + h] : 0.0f;
    const float r1 = p.logdist && live ? p.logdist[h0 + h] : 0.0f, r2 = p.logdist && live ? p.logdist[p.heads + h0 + h] : 0.0f;
    float m = -INFINITY, l = 0.0f, o[kTiles][2];          // first and third terms' sums together, or the second ones'
#pragma unroll
    for (int i = 0; i < kTiles; ++i) o[i][0] = o[i][1] = 0.0f;
    // ldmatrix rows: keys as they lie (two key tiles x two halves of a k-step), values transposed (two value tiles x two halves of the keys)
    const uint32_t k_at = (((lane & 7) + (lane & 16 ? 8 : 0)) * D * 2) | (((lane & 8 ? 1 : 0) ^ (lane & 7)) << 4);
    const uint32_t v_at = ((kRun + (lane & 15)) * D * 2) | (((lane & 16 ? 1 : 0) ^ (lane & 7)) << 4);
    // Several terms times an infinite value are no number, where the fp32 product would be infinite: a warp whose sums come out like that walks its runs once
    // more with the later terms' products left out wherever they are not finite. The first terms then give what fp32 gives.
    auto finite = [](float x) { return fabsf(x) <= 3.402823466e38f ? x : 0.0f; };
    auto walk = [&](auto careful_) {
        constexpr bool careful = decltype(careful_)::value;
        int stage = 0;
        for (int run = first_run; run < n_runs; run += workers) {
            cp_async_wait<kRing - 2>();
            __syncwarp();
            const int j0 = first_key(run);
            const uint32_t base = ring + stage * Tile::kStage * 2;
            float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int ks = 0; ks < kSteps; ks += 2) {
                float part[2][4];
                uint32_t ka[4], kb[4];
                ldmatrix4(ka, base + (k_at ^ (ks * 32)));
                ldmatrix4(kb, base + (k_at ^ ((ks + 1) * 32)));
                mma_bf16_zero(part[0], qa[ks], ka[0], ka[1]);
                mma_bf16_zero(part[1], qa[ks], ka[2], ka[3]);
                mma_bf16_16816(part[0], qa[ks + 1], kb[0], kb[1]);
                mma_bf16_16816(part[1], qa[ks + 1], kb[2], kb[3]);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[i][e] += part[i][e];
            }
            // first + third term here, the second on the neighbouring lane: both then hold the head's scores of keys 2c, 2c + 1 (+ 8)
            float w[4], mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float here = s[i >> 1][i & 1], third = s[i >> 1][2 + (i & 1)];
                const float mine = careful ? (second ? finite(here) : here) + finite(third) : here + third;
                w[i] = mine + __shfl_xor_sync(0xffffffffu, mine, 4);
                w[i] = kOpts ? seq_score(w[i], p.scale, p.softcap, slope, r1, r2, pos, j0 + (i >> 1) * 8 + 2 * c + (i & 1)) : w[i] * p.scale;
            }
            if (j0 + kRun - 1 > pos || (pos - j0 >= wnd && j0 + kRun > p.keep_first)) {      // some key of the run is hidden
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (!seq_sees(pos, j0 + (i >> 1) * 8 + 2 * c + (i & 1), wnd, p.keep_first)) w[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) mx = fmaxf(mx, w[i]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float mn = fmaxf(m, mx);
            if (__any_sync(0xffffffffu, mn != m)) {
                const float corr = mn == -INFINITY ? 1.0f : expf(m - mn);
                l *= corr;
#pragma unroll
                for (int i = 0; i < kTiles; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) o[i][e] *= corr;
                m = mn;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                w[i] = w[i] == -INFINITY ? 0.0f : expf(w[i] - mn);
                l += w[i];
            }
            uint32_t pa[4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t t1, t2, t3;
                split3_bf16(w[half * 2], w[half * 2 + 1], t1, t2, t3);
                pa[half * 2] = second ? t2 : t1;
                pa[half * 2 + 1] = second ? 0u : t3;
            }
#pragma unroll
            for (int nt = 0; nt < kTiles; nt += 2) {
                uint32_t vb[4];
                ldmatrix4_trans(vb, base + (v_at ^ (nt * 16)));
                float part[2][4];
                mma_bf16_zero(part[0], pa, vb[0], vb[1]);
                mma_bf16_zero(part[1], pa, vb[2], vb[3]);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) o[nt + i][e] += careful ? (second ? finite(part[i][e]) : part[i][e]) + finite(part[i][2 + e]) : part[i][e] + part[i][2 + e];
            }
            __syncwarp();                       // every lane has read the stage that is filled next
            issue(run + (kRing - 1) * workers, stage == 0 ? kRing - 1 : stage - 1);
            stage = stage + 1 == kRing ? 0 : stage + 1;
        }
    };
    walk(std::false_type{});
    bool wild = false;
#pragma unroll
    for (int i = 0; i < kTiles; ++i) wild |= o[i][0] != o[i][0] || o[i][1] != o[i][1];
    if (__any_sync(0xffffffffu, wild)) {
        cp_async_wait<0>();
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kRing - 1; ++i) issue(first_run + i * workers, i);
        m = -INFINITY;
        l = 0.0f;
#pragma unroll
        for (int i = 0; i < kTiles; ++i) o[i][0] = o[i][1] = 0.0f;
        walk(std::true_type{});
    }
    // The terms' results meet on neighbouring lanes: the lane of the first and third terms keeps the first half of the columns, the other the second.
    float v[kTiles / 2][2];
#pragma unroll
    for (int i = 0; i < kTiles / 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float lo = o[i][e], hi = o[i + kTiles / 2][e];
            v[i][e] = (second ? hi : lo) + __shfl_xor_sync(0xffffffffu, second ? lo : hi, 4);
        }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    // every CTA of the cluster gets the sums of its own share of the results, and everybody's maxima
    const int share = (G * D + 2 * CS - 1) / (2 * CS) * 2, worker = rank * kDecodeWarps + warp, columns = G * D;
    if (!alone) cluster.barrier_wait();
    if (live) {
#pragma unroll
        for (int i = 0; i < kTiles / 2; ++i) {
            const int at = h * D + (second ? D / 2 : 0) + i * 8 + 2 * c, to = at / share;
            *reinterpret_cast<float2*>(cluster.map_shared_rank(got_o, base_rank + to) + worker * share + at % share) = make_float2(v[i][0], v[i][1]);
        }
        if (!second)
            for (int r = c; r < CS; r += 4) cluster.map_shared_rank(got_ml, base_rank + r)[worker * 4 + h] = make_float2(m, l);
    }
    if (alone) __syncthreads(); else cluster.sync();
    if (warp < G) {
        const int n = CS * kDecodeWarps;
        float M = -INFINITY, L = 0.0f;
        for (int i = lane; i < n; i += 32) M = fmaxf(M, got_ml[i * 4 + warp].x);
        M = warp_max(M);
        for (int i = lane; i < n; i += 32) {
            const float2 ml = got_ml[i * 4 + warp];
            const float f = ml.x == -INFINITY ? 0.0f : expf(ml.x - M);
            weight[i][warp] = f;
            L = fmaf(ml.y, f, L);
        }
        L = warp_sum(L);
        if (lane == 0) {
            total[warp][0] = M;
            total[warp][1] = L;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < share; i += kDecodeWarps * 32) {
        const int at = rank * share + i, hh = at / D, col = at % D;
        if (at >= columns) break;
        float sums[kDecodeWarps] = {};                  // (several: fewer roundings in a row)
#pragma unroll 4
        for (int wkr = 0; wkr < CS * kDecodeWarps; wkr += kDecodeWarps)
#pragma unroll
            for (int e = 0; e < kDecodeWarps; ++e) sums[e] = fmaf(got_o[(wkr + e) * share + i], weight[wkr + e][hh], sums[e]);
        float acc = (sums[0] + sums[1]) + (sums[2] + sums[3]);
        if (p.out || p.out16) {
            acc *= 1.0f / total[hh][1];
            if (p.out) p.out[(size_t)t * p.ldo + (size_t)(h0 + hh) * D + col] = acc;
            if (p.out16) p.out16[((size_t)t * p.heads + h0 + hh) * D + col] = f32_to_bf16_bits(acc);
        } else {
            float* rec = p.ws + (((size_t)t * p.heads + h0 + hh) * p.nsplit + split) * (D + 2);
            rec[2 + col] = acc;
            if (col == 0) {
                rec[0] = total[hh][0];
                rec[1] = total[hh][1];
            }
        }
    }
    }
}

#endif

}  // namespace sllm
