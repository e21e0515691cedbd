// csrc/seq_attn_decode.cuh — attention of steps of single tokens (decoding) over the paged cache; part of seq_attn.cu.
#pragma once
#include <cooperative_groups.h>

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
};

#ifdef __CUDACC__

__device__ __forceinline__ float seq_score(float dot, float scale, float softcap, float slope, float r1, float r2, int qpos, int key) {
    float sc = dot * scale;
    if (softcap > 0.0f) sc = softcap * tanhf(sc / softcap);
    sc -= slope * (float)(qpos - key);
    if (r1 != 0.0f) sc -= r1 * log1pf(r2 * (float)(qpos - key));
    return sc;
}

// 16 bytes of a cache row as pairs of floats
__device__ __forceinline__ void cache_pairs(const uint4& u, uint64_t (&p)[4], const uint16_t*) {
    p[0] = pair_f32(u.x << 16, u.x & 0xffff0000u);
    p[1] = pair_f32(u.y << 16, u.y & 0xffff0000u);
    p[2] = pair_f32(u.z << 16, u.z & 0xffff0000u);
    p[3] = pair_f32(u.w << 16, u.w & 0xffff0000u);
}
__device__ __forceinline__ void cache_pairs(const uint4& u, uint64_t (&p)[2], const float*) {
    p[0] = pair_f32(u.x, u.y);
    p[1] = pair_f32(u.z, u.w);
}

constexpr int kDecodeWarps = 4, kDecodeCluster = 16;     // warps of a CTA, CTAs of a cluster at most

// One query per sequence: G query heads of one kv head against that head's cache rows. Bound: HBM (each row is read once and used G times), so
// rows go from global memory to registers and nothing is staged: eight lanes share a row (16-byte loads, neighbours next to each other), the four
// groups of lanes of a warp hold neighbouring rows, kSteps of them in flight per lane, values requested before the scores are worked on. Everything
// is fp32 (queries as they are, two products per instruction); G x kSteps scores cross the eight lanes in one halving exchange, which leaves
// every score on one lane for its exponential. A sequence's rows are dealt in runs of 4 x kSteps keys to all warps of a thread-block cluster, so that
// the longest context of a step is spread over up to 16 CTAs whatever the step's share count; every warp sends its sums to the CTAs that own the
// columns (distributed shared memory, one barrier), which merge them and write the result (or one record per share when something still follows).
template <typename KV, int KL, int VL, int G, int kSteps>     // 16-byte loads per lane of a key / value row: dk = 8 * KL * E, dv = 8 * VL * E
__global__ void __launch_bounds__(kDecodeWarps * 32) seq_attention_decode_kernel(AttnArgs p) {
    namespace cg = cooperative_groups;
    constexpr int E = 16 / sizeof(KV), PE = E / 2, dk = 8 * KL * E, dv = 8 * VL * E, VAL = G * kSteps;
    constexpr int kPer = VAL >= 8 ? VAL / 8 : 1, kDup = VAL >= 8 ? 1 : 8 / VAL;      // scores per lane after the exchange, lanes that hold the same one
    constexpr int kRun = 4 * kSteps;                                                  // keys of one step of a warp
    static_assert(kBK % kRun == 0, "a run of keys lies inside one tile");
    constexpr int kPairs = G * VL * PE;                  // pairs of sums a lane keeps
    // what the cluster's warps send this CTA: their sums for its share of the G * dv results, and every warp's (maximum, sum) per head
    __shared__ __align__(16) float got_o[kDecodeWarps * G * dv];
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
    const KV* kp = reinterpret_cast<const KV*>(p.k_pool);
    const KV* vp = reinterpret_cast<const KV*>(p.v_pool);
    const int32_t* table = b.block_table + (size_t)slot * b.max_pages;

    uint64_t qv[G][KL * PE];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < KL; ++i) {
            const float* src = p.q + (size_t)t * p.ldq + (size_t)(h0 + g) * dk + (i * 8 + j8) * E;
#pragma unroll
            for (int e = 0; e < PE; ++e) qv[g][i * PE + e] = pair_f32(src[2 * e], src[2 * e + 1]);
        }
    // this lane's scores: head og, steps os .. os + kPer - 1 of its group's keys
    const int og = (j8 / kDup) * kPer / kSteps, os = (j8 / kDup) * kPer % kSteps;
    const float slope = p.slopes ? p.slopes[h0 + og] : 0.0f;
    const float r1 = p.logdist ? p.logdist[h0 + og] : 0.0f, r2 = p.logdist ? p.logdist[p.heads + h0 + og] : 0.0f;
    float m[G], l = 0.0f;                       // running maxima (all lanes alike); this lane's share of the sum of head og
    uint64_t acc[G][VL * PE];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY;
#pragma unroll
        for (int i = 0; i < VL * PE; ++i) acc[g][i] = 0ull;
    }
    auto first_key = [&](int run) { return tiles.tile_of(run / kRuns) * kBK + run % kRuns * kRun; };
    // rows the sequence does not have yet read as zeros (their memory may hold anything)
    auto load_keys = [&](uint4 (&u)[kSteps][KL], int j0, int page) {
        const KV* row = kp + seq_pool_row(page, p.kv_heads, gkv, b.page_len, j0 % b.page_len + kg, dk) + j8 * E;
#pragma unroll
        for (int s = 0; s < kSteps; ++s)
#pragma unroll
            for (int i = 0; i < KL; ++i) u[s][i] = j0 + 4 * s + kg <= pos ? ldg_stream(row + (size_t)(4 * s) * dk + i * 8 * E) : make_uint4(0u, 0u, 0u, 0u);
    };
    auto load_values = [&](uint4 (&u)[kSteps][VL], int j0, int page) {
        const KV* row = vp + seq_pool_row(page, p.kv_heads, gkv, b.page_len, j0 % b.page_len + kg, dv) + j8 * E;
#pragma unroll
        for (int s = 0; s < kSteps; ++s)
#pragma unroll
            for (int i = 0; i < VL; ++i) u[s][i] = j0 + 4 * s + kg <= pos ? ldg_stream(row + (size_t)(4 * s) * dv + i * 8 * E) : make_uint4(0u, 0u, 0u, 0u);
    };
    // A run's keys are asked for as soon as the previous run's have been multiplied, its values likewise: one of the two is always on its way.
    uint4 ku[kSteps][KL], vu[kSteps][VL];
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
            for (int i = 0; i < KL; ++i) {
                uint64_t kk[PE];
                cache_pairs(ku[s][i], kk, kp);
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
                for (int i = 0; i < VL * PE; ++i) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[g][i]) : "l"(c2));
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
            for (int i = 0; i < VL; ++i) {
                uint64_t vv[PE];
                cache_pairs(vu[s][i], vv, vp);
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
    for (int i = 0; i < kPairs; ++i) v[i] = acc[i / (VL * PE)][i % (VL * PE)];
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
    const int share = G * dv / CS, worker = rank * kDecodeWarps + warp;
    cluster.barrier_wait();
#pragma unroll
    for (int i = 0; i < kPairs / 4; ++i) {
        const int at = kg * (kPairs / 4) + i, g = at / (VL * PE), r = at % (VL * PE);
        const int item = g * dv + (r / PE * 8 + j8) * E + r % PE * 2, to = item / share;
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
        float M = -INFINITY, L = 0.0f;
        for (int i = lane; i < n; i += 32) M = fmaxf(M, got_ml[i][warp].x);
        M = warp_max(M);
        for (int i = lane; i < n; i += 32) {
            const float f = got_ml[i][warp].x == -INFINITY ? 0.0f : expf(got_ml[i][warp].x - M);
            weight[i][warp] = f;
            L = fmaf(got_ml[i][warp].y, f, L);
        }
        L = warp_sum(L);
        if (lane == 0) {
            total[warp][0] = M;
            total[warp][1] = L;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < share; i += kDecodeWarps * 32) {
        const int item = rank * share + i, g = item / dv, c = item % dv;
        float o = 0.0f;
#pragma unroll 4
        for (int w = 0; w < CS * kDecodeWarps; ++w) o = fmaf(got_o[w * share + i], weight[w][g], o);
        if (p.out || p.out16) {
            o *= 1.0f / total[g][1];
            if (p.out) p.out[(size_t)t * p.ldo + (size_t)(h0 + g) * dv + c] = o;
            if (p.out16) p.out16[((size_t)t * p.heads + h0 + g) * dv + c] = f32_to_bf16_bits(o);
        } else {
            float* rec = p.ws + (((size_t)t * p.heads + h0 + g) * p.nsplit + split) * (dv + 2);
            rec[2 + c] = o;
            if (c == 0) {
                rec[0] = total[g][0];
                rec[1] = total[g][1];
            }
        }
    }
}

#endif

}  // namespace sllm
