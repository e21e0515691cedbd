// csrc/seq_chunk.cu — the delta rule (decay per head or per key channel) and linear attention with a constant decay, in blocks of 32 tokens
// on the tensor cores: portions of prompts in bf16 mode. Within a block that starts from the state S0 [dk][dv], with G_i the running sum of
// the logarithms of the decays (a vector over the key channels) up to token i,
//     u_i = beta_i (v_i - S0^T (e^G_i k_i) - sum_{j<i} A_ij u_j),       A_ij = sum_c k_ic k_jc e^(G_ic - G_jc)
//     o_i = S0^T (e^G_i q_i) + sum_{j<=i} B_ij u_j,                     B_ij = sum_c q_ic k_jc e^(G_ic - G_jc)
//     S'  = e^G_n S0 + sum_j (e^(G_n - G_j) k_j) u_j^T
// (e^G per key channel, i.e. on the rows of S). The u of a block solve a 32 x 32 triangular system, u = M (v - S0^T (e^G k)); linear attention
// is the case M = 1, no S0 term in u. No factor exceeds 1: a difference of sums is formed before its exponential. The sums start anew at a block's middle, so that they stay as
// small, and their differences as exact, as over 16 tokens.
//
// (1) seq_chunk_prepare_kernel, CTA = (block, head), all blocks of the step in parallel: silu / rotation / unit vectors, G, A and B (fp32, 4 x 4 entries and an eighth of the channels
// per thread), M from the inverses of its two 16 x 16 triangles; leaves e^G k, e^G q, e^(G_n - G) k, M and B as the tensor-core fragments the walk
// will load, each as two bf16 terms (x = hi + lo, |x - hi - lo| <= 2^-17 |x|), and e^G_n in fp32. Bound: shared memory's bandwidth and the exponentials: decays that are one number per
// head multiply finished sums and whole rows (2048 tokens of 16 heads: 58 us with the decays inside the sums and blocks of 16 in two threads per entry, 42 like this).
// (2) seq_chunk_walk_kernel, CTA = (portion, head, 16 or 32 value columns), two or four warps = 16 value columns, a share of the key channels each: their part of
// S^T [16][dk] stays in the accumulators (fp32) from the portion's first token to its last. An accumulator fragment is register for register
// an A fragment of the next product, so state and u never leave the registers; all products take both operands as two bf16 terms (three products, four where u is an operand, fp32 accumulation), which keeps
// the recurrence at fp32 working accuracy (against float64 in the mean over 120 shapes and decays 0.78 of the error of blocks of 16 without the products of second terms, in none more). The blocks' records arrive by one bulk copy each, three stages. Bound: latency of a block's chain (products with the state, their exchange
// between the warps, u, the state); a block of 32 takes hardly longer than one of 16 (2048 tokens of 16 heads: 1.05 us for 16, 1.6 for 32, a walk 137 | 103 us). Where blocks of 16 are
// ahead all the same, the kernels of seq_chunk16.cu run (chunk_in_16).
#include "seq_chunk.cuh"
#include "mega_common.cuh"

namespace sllm {

constexpr int kPrepThreads = 288;    // eight threads per 4 x 4 entries of a triangle of 32 x 32
constexpr int kWalkStages = 3;

struct ChunkPlace { int seg, start, n, id; };      // segment, first token in the batch, tokens, number of the block in segment order
__device__ __forceinline__ ChunkPlace chunk_place(const sllm_seq_batch& b, int tile) {
    ChunkPlace c;
    c.seg = b.qt_seg[tile];
    const int off = b.qt_off[tile];
    c.n = min(kChunk, b.seg_len[c.seg] - off);
    c.start = b.seg_start[c.seg] + off;
    c.id = b.seg_tile0[c.seg] + off / kChunk;
    return c;
}

__device__ __forceinline__ float4 chunk_scale(const float4& a, const float4& e) { return make_float4(a.x * e.x, a.y * e.y, a.z * e.z, a.w * e.w); }
__device__ __forceinline__ float4 chunk_decay(const float4& a, const float4& b) { return make_float4(exp2f(a.x - b.x), exp2f(a.y - b.y), exp2f(a.z - b.z), exp2f(a.w - b.w)); }
__device__ __forceinline__ float chunk_dot(const float4& a, const float4& b, float c) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c)))); }

// lanes with `bit` set keep (and complete) the upper half of 2 K values, the others the lower half
template <int K, int N>
__device__ __forceinline__ void chunk_halve(float (&v)[N], bool up, int bit) {
#pragma unroll
    for (int x = 0; x < K; ++x) {
        const float give = up ? v[x] : v[x + K], keep = up ? v[x + K] : v[x];
        v[x] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
}

enum { kDecayConstant = 0, kDecayHead = 1, kDecayChannel = 2 };      // linear attention; the delta rule with one decay per head, per key channel
template <int kMode, int dkp> struct ChunkPrepShared {               // floats
    static constexpr int ld = dkp + 8, kRows = kChunk * ld, kTri = kChunk * (kChunk + 1);
    static constexpr int kBytes = ((kMode == kDecayChannel ? 3 : 2) * kRows + (kMode == kDecayConstant ? 1 : 3) * kTri + 16 * 17) * 4;
};

// vec: rows of q, k, v (and of the channels' steps) may be read 16 bytes at a time
template <int kMode, int dkp>
__global__ void __launch_bounds__(kPrepThreads, kMode == kDecayChannel ? 2 : 3) seq_chunk_prepare_kernel(ChunkArgs p, int vec) {
    constexpr bool kDelta = kMode != kDecayConstant, kChannel = kMode == kDecayChannel;
    using Sh = ChunkPrepShared<kMode, dkp>;
    constexpr int ld = Sh::ld, H = kChunk / 2;
    extern __shared__ __align__(16) float cp_sm[];
    __shared__ float s_beta[kChunk], s_g[kChunk], s_pre[kChunk], s_end[kChunk];
    const sllm_seq_batch& b = p.b;
    const ChunkPlace c = chunk_place(b, blockIdx.x);
    if (c.n <= 0) return;
    const int h = blockIdx.y, kvh = h / (p.heads / p.kv_heads), dk = p.dk;
    float* s_k = cp_sm;                             // [32][ld]
    float* s_q = s_k + Sh::kRows;                   // [32][ld]
    float* s_G = s_q + Sh::kRows;                   // [32][ld], a decay per channel only: sums of a half
    float (*s_B)[kChunk + 1] = reinterpret_cast<float (*)[kChunk + 1]>(s_q + (kChannel ? 2 : 1) * Sh::kRows);
    float (*s_A)[kChunk + 1] = s_B + kChunk;        // the delta rule only
    float (*s_M)[kChunk + 1] = s_A + kChunk;
    float (*s_T)[17] = reinterpret_cast<float (*)[17]>(s_M + kChunk);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float rate = kDelta ? expf(p.A_log[h]) : p.rate[h];
    const float lg = -rate * kLog2e;    // constant decay: its base-2 logarithm
    auto load4 = [&](const float* row, int ch, bool has) {             // channels ch .. ch + 3 of a row, zeros beyond the head
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!has) return v;
        if (vec && ch < dk) return *reinterpret_cast<const float4*>(row + ch);
        if (ch < dk) v.x = row[ch];
        if (ch + 1 < dk) v.y = row[ch + 1];
        if (ch + 2 < dk) v.z = row[ch + 2];
        if (ch + 3 < dk) v.w = row[ch + 3];
        return v;
    };
    auto silu4 = [](float4 v) { return make_float4(v.x * seq_sigmoid(v.x), v.y * seq_sigmoid(v.y), v.z * seq_sigmoid(v.z), v.w * seq_sigmoid(v.w)); };
    // all of a thread's rows are asked for before the first of them is worked on
    constexpr int kWords = kChunk * dkp / 4, kRounds = (kWords + kPrepThreads - 1) / kPrepThreads;
    {
        float4 kv[kRounds], qv[kRounds], a[kRounds], bias[kRounds];
#pragma unroll
        for (int x = 0; x < kRounds; ++x) {
            const int i = threadIdx.x + x * kPrepThreads, tok = i / (dkp / 4), ch = (i % (dkp / 4)) * 4;
            const bool has = i < kWords && tok < c.n;
            const size_t t = (size_t)(c.start + (has ? tok : 0));
            kv[x] = load4(p.k + t * p.ldk + (size_t)kvh * dk, ch, has);
            qv[x] = load4(p.q + t * p.ldq + (size_t)kvh * dk, ch, has);
            if (kChannel) {
                a[x] = load4(p.al + t * p.lda + (size_t)h * dk, ch, has);
                bias[x] = load4(p.dt_bias + (size_t)h * dk, ch, has);
            }
        }
#pragma unroll
        for (int x = 0; x < kRounds; ++x) {
            const int i = threadIdx.x + x * kPrepThreads, tok = i / (dkp / 4), ch = (i % (dkp / 4)) * 4;
            if (i >= kWords) break;
            if (!kDelta && p.silu) {
                kv[x] = silu4(kv[x]);
                qv[x] = silu4(qv[x]);
            }
            *reinterpret_cast<float4*>(s_k + tok * ld + ch) = kv[x];
            *reinterpret_cast<float4*>(s_q + tok * ld + ch) = qv[x];
            if (kChannel) {
                const bool has = tok < c.n;
                *reinterpret_cast<float4*>(s_G + tok * ld + ch) =
                    make_float4(has && ch < dk ? lg * seq_softplus(a[x].x + bias[x].x) : 0.0f, has && ch + 1 < dk ? lg * seq_softplus(a[x].y + bias[x].y) : 0.0f,
                                has && ch + 2 < dk ? lg * seq_softplus(a[x].z + bias[x].z) : 0.0f, has && ch + 3 < dk ? lg * seq_softplus(a[x].w + bias[x].w) : 0.0f);
            }
        }
    }
    if (!kDelta && p.silu)                               // the values too, for the walk
        for (int tok = warp; tok < c.n; tok += kPrepThreads / 32) {
            const float* src = p.v + (size_t)(c.start + tok) * p.ldv + (size_t)h * p.dv;
            float* dst = p.v_ws + ((size_t)c.id * kChunk + tok) * p.heads * p.dv + (size_t)h * p.dv;
            if (vec)
                for (int j = 4 * lane; j < p.dv; j += 128) *reinterpret_cast<float4*>(dst + j) = silu4(*reinterpret_cast<const float4*>(src + j));
            else
                for (int j = lane; j < p.dv; j += 32) dst[j] = src[j] * seq_sigmoid(src[j]);
        }
    if (kDelta && warp == 8) {
        const bool has = lane < c.n;
        s_beta[lane] = has ? seq_sigmoid(p.bl[(size_t)(c.start + lane) * p.ldb + h]) : 0.0f;
        if (!kChannel) {                                 // sums over either half, one token behind the other
            const float g = has ? lg * seq_softplus(p.al[(size_t)(c.start + lane) * p.lda + h] + p.dt_bias[h]) : 0.0f;
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const float x = __shfl_sync(0xffffffffu, g, (lane & H) + i);
                if (i <= lane % H) sum += x;
            }
            const float first = __shfl_sync(0xffffffffu, sum, H - 1), second = __shfl_sync(0xffffffffu, sum, kChunk - 1);
            s_g[lane] = sum;
            s_pre[lane] = exp2f(lane < H ? sum : first + sum);
            s_end[lane] = exp2f(lane < H ? (first - sum) + second : second - sum);
        }
    }
    const int last = c.n - 1;
    if (!kDelta && warp == 8) {
        s_pre[lane] = exp2f(lg * (float)(min(lane, last) + 1));
        s_end[lane] = exp2f(lg * (float)(last - min(lane, last)));
    }
    __syncthreads();
    for (int tok = warp; tok < c.n; tok += kPrepThreads / 32) {
        float* kr = s_k + tok * ld;
        float* qr = s_q + tok * ld;
        if (kDelta) {                                    // unit vectors
            float sk = 0.0f, sq = 0.0f;
            for (int ch = lane; ch < dk; ch += 32) {
                sk = fmaf(kr[ch], kr[ch], sk);
                sq = fmaf(qr[ch], qr[ch], sq);
            }
            const float ik = 1.0f / sqrtf(warp_sum(sk) + p.unit_eps), iq = p.scale / sqrtf(warp_sum(sq) + p.unit_eps);
            for (int ch = lane; ch < dk; ch += 32) {
                kr[ch] *= ik;
                qr[ch] *= iq;
            }
        } else {
            for (int i = lane; i < p.n_freq; i += 32) {
                const int ia = p.layout == 0 ? 2 * i : i, ib = p.layout == 0 ? 2 * i + 1 : i + p.n_freq;
                const float2 a = p.angles[(size_t)(c.start + tok) * p.n_freq + i];
                const float ku = kr[ia], kw = kr[ib], qu = qr[ia], qw = qr[ib];
                kr[ia] = ku * a.x - kw * a.y;
                kr[ib] = kw * a.x + ku * a.y;
                qr[ia] = qu * a.x - qw * a.y;
                qr[ib] = qw * a.x + qu * a.y;
            }
            __syncwarp();
            if (p.scale != 1.0f)
                for (int ch = lane; ch < dk; ch += 32) kr[ch] *= p.scale;
        }
    }
    if (kChannel && (int)threadIdx.x < 2 * dkp) {        // running sums of a half (a column no other thread touches)
        float* col = s_G + (threadIdx.x / dkp) * H * ld + threadIdx.x % dkp;
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < H; ++i) {
            sum += col[i * ld];
            col[i * ld] = sum;
        }
    }
    __syncthreads();
    // The two matrices: eight threads per 4 x 4 entries (rows ti, columns tj <= ti), each every eighth group of four channels. The sums of A and B change lanes in a halving
    // exchange, after which a lane has N / 8 of them.
    {
        constexpr int N = kDelta ? 32 : 16;
        const int e = threadIdx.x >> 3, kg = threadIdx.x & 7;
        int ti = 0;
        while ((ti + 1) * (ti + 2) / 2 <= e) ++ti;
        const int tj = e - ti * (ti + 1) / 2;
        const float *ki = s_k + 4 * ti * ld, *kj = s_k + 4 * tj * ld, *qi = s_q + 4 * ti * ld, *Gi = s_G + 4 * ti * ld, *Gj = s_G + 4 * tj * ld;
        const bool cross = ti >= H / 4 && tj < H / 4;
        float v[N];
#pragma unroll
        for (int x = 0; x < N; ++x) v[x] = 0.0f;
        auto at = [](const float* row, int ch) { return *reinterpret_cast<const float4*>(row + ch); };
        for (int ch = 4 * kg; ch < dkp; ch += 32) {
            float4 x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = at(kj + j * ld, ch);
            if (kChannel && ti != tj) {                  // decays from token j to the end of the first half, or to the tile's first row; from there on to token i
                const float4 to = cross ? at(s_G + (H - 1) * ld, ch) : at(Gi, ch);
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = chunk_scale(x[j], chunk_decay(to, at(Gj + j * ld, ch)));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 y = at(qi + i * ld, ch), z = y;
                if (kDelta) z = at(ki + i * ld, ch);
                if (kChannel) {
                    const float4 g = at(Gi + i * ld, ch);
                    if (ti != tj) {
                        const float4 f = chunk_decay(g, cross ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : at(Gi, ch));
                        y = chunk_scale(y, f);
                        z = chunk_scale(z, f);
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (j > i) continue;
                            const float4 f = chunk_scale(x[j], chunk_decay(g, at(Gj + j * ld, ch)));
                            v[4 * i + j] = chunk_dot(z, f, v[4 * i + j]);
                            v[N - 16 + 4 * i + j] = chunk_dot(y, f, v[N - 16 + 4 * i + j]);
                        }
                        continue;
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (kDelta) v[4 * i + j] = chunk_dot(z, x[j], v[4 * i + j]);
                    v[N - 16 + 4 * i + j] = chunk_dot(y, x[j], v[N - 16 + 4 * i + j]);
                }
            }
        }
        chunk_halve<N / 2>(v, lane & 4, 4);
        chunk_halve<N / 4>(v, lane & 2, 2);
        chunk_halve<N / 8>(v, lane & 1, 1);
#pragma unroll
        for (int x = 0; x < N / 8; ++x) {
            const int idx = (lane & 7) * (N / 8) + x, i = 4 * ti + idx / 4 % 4, j = 4 * tj + idx % 4;
            float w = v[x];
            if (kMode == kDecayConstant) w *= exp2f(lg * (float)(i - j));
            if (kMode == kDecayHead) w *= exp2f(i >= H && j < H ? s_g[i] + (s_g[H - 1] - s_g[j]) : s_g[i] - s_g[j]);
            if (kDelta && idx < 16) {
                s_A[i][j] = w;
            } else {
                s_B[i][j] = i >= j ? w : 0.0f;
                if (ti != tj) s_B[j][i] = 0.0f;
            }
        }
    }
    __syncthreads();
    uint8_t* rec = p.ws + ((size_t)c.id * p.heads + h) * chunk_record_bytes(dkp);
    constexpr size_t plane = (size_t)kChunk * dkp * 2;
    uint8_t* mats = rec + 6 * plane;                     // M hi, M lo, B hi, B lo: the 16 x 16 blocks (0, 0), (1, 0) and (1, 1) of each, 512 bytes a block
    float* D = reinterpret_cast<float*>(mats + 12 * 512);
    if (kDelta && warp < 2) {                            // M = (1 + diag(beta) A)^-1 diag(beta) of either half, lane = column
        const int o = warp * H;
        float m[H];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            float acc = 0.0f;
#pragma unroll
            for (int l = 0; l < i; ++l) acc = fmaf(s_A[o + i][o + l], m[l], acc);
            m[i] = s_beta[o + i] * ((i == lane ? 1.0f : 0.0f) - acc);
            if (lane < H) s_M[o + i][o + lane] = m[i];
        }
    }
    // the decay from the block's start to after token i, and from after token i to the block's end
    auto before = [&](int i, int ch) { return !kChannel ? s_pre[i] : exp2f(i < H ? s_G[i * ld + ch] : s_G[(H - 1) * ld + ch] + s_G[i * ld + ch]); };
    auto behind = [&](int i, int ch) {
        if (!kChannel) return s_end[i];
        return exp2f(i < H ? (s_G[(H - 1) * ld + ch] - s_G[i * ld + ch]) + s_G[(kChunk - 1) * ld + ch] : s_G[(kChunk - 1) * ld + ch] - s_G[i * ld + ch]);
    };
    constexpr int granules = dkp * 4;                    // 16-byte pieces of a plane: [half of the tokens][k-step of channels][lane]
    for (int x = threadIdx.x + (kDelta ? 0 : granules); x < 3 * granules; x += kPrepThreads) {     // (without a correction there is no S0 term in u)
        const int which = x / granules, at = x % granules, pr = at / (granules / 2), ks = (at >> 5) % (dkp / 16), gr = (at & 31) >> 2, cc = at & 3;
        float v[8];
#pragma unroll
        for (int y = 0; y < 4; ++y) {                    // pairs: (first / second group of 8) x (first / second half of the k-step)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int outer = (y >> 1) * 8 + gr, inner = (y & 1) * 8 + 2 * cc + half;
                if (which < 2) {
                    const int tok = pr * H + outer, ch = ks * 16 + inner;
                    v[2 * y + half] = (which == 0 ? s_k : s_q)[tok * ld + ch] * before(tok, ch);
                } else {
                    const int tok = pr * H + inner, ch = ks * 16 + outer;
                    v[2 * y + half] = s_k[tok * ld + ch] * behind(tok, ch);
                }
            }
        }
        chunk_put(rec + 2 * which * plane, rec + (2 * which + 1) * plane, at, v);
    }
    for (int ch = threadIdx.x; ch < dkp; ch += kPrepThreads) D[ch] = before(kChannel ? kChunk - 1 : last, ch);
    if (kDelta) {                                        // the block (1, 0) of M: -M(1,1) A(1,0) M(0,0)
        __syncthreads();
        const int i = threadIdx.x / H, j = threadIdx.x % H;
        if (i < H) {
            float acc = 0.0f;
#pragma unroll
            for (int l = 0; l < H; ++l) acc = fmaf(s_A[H + i][l], l >= j ? s_M[l][j] : 0.0f, acc);
            s_T[i][j] = acc;
        }
        __syncthreads();
        if (i < H) {
            float acc = 0.0f;
#pragma unroll
            for (int l = 0; l < H; ++l) acc = fmaf(l <= i ? s_M[H + i][H + l] : 0.0f, s_T[l][j], acc);
            s_M[H + i][j] = -acc;
        }
        __syncthreads();
    }
    for (int x = threadIdx.x + (kDelta ? 0 : 96); x < 192; x += kPrepThreads) {
        const int which = x / 96, blk = (x >> 5) % 3, i0 = blk > 0 ? H : 0, j0 = blk > 1 ? H : 0, gr = (x & 31) >> 2, cc = x & 3;
        float v[8];
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = i0 + (y >> 1) * 8 + gr, j = j0 + (y & 1) * 8 + 2 * cc + half;
                v[2 * y + half] = which == 0 ? s_M[i][j] : s_B[i][j];
            }
        chunk_put(mats + (2 * which * 3 + blk) * 512, mats + ((2 * which + 1) * 3 + blk) * 512, x & 31, v);
    }
}

// KS: k-steps of 16 key channels. PARTS warps share 16 value columns, each owning KS / PARTS of the k-steps; they add their parts of the
// products with the old state through shared memory and finish 32 / PARTS tokens each. GROUPS: how many times 16 columns a CTA takes.
template <int KS, int PARTS, int GROUPS, bool kDelta>
__global__ void __launch_bounds__(PARTS * GROUPS * 32, 1) seq_chunk_walk_kernel(ChunkArgs p, int vec) {
    extern __shared__ __align__(16) uint8_t cw_sm[];
    __shared__ uint64_t landed[kWalkStages];             // the records
    constexpr int dkp = KS * 16, HS = KS / PARTS, kThreads = PARTS * GROUPS * 32, kCols = GROUPS * 16, kTiles = kChunk / 8;
    constexpr bool kThird = kDelta && KS == 2;           // u as three bf16 terms
    constexpr uint32_t kPlane = kChunk * dkp * 2;
    constexpr uint32_t rec_bytes = (uint32_t)chunk_record_bytes(dkp), stage_bytes = rec_bytes + kChunk * kCols * 4;
    const sllm_seq_batch& b = p.b;
    const int seg = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * kCols;
    const int start = b.seg_start[seg], len = b.seg_len[seg], slot = b.seg_slot[seg];
    const int blocks = (len + kChunk - 1) / kChunk;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    const int group = warp % GROUPS, part = warp / GROUPS, k0 = part * HS;   // this warp's value columns and first k-step
    const int cl = group * 16 + g, r0 = col0 + cl, r1 = r0 + 8;              // this thread's two value columns
    const bool ok0 = r0 < p.dv, ok1 = r1 < p.dv;
    // what the warps of a group hand each other: [group][part][x of four tiles of 8 tokens, o of four][lane]
    float4* exchange = reinterpret_cast<float4*>(cw_sm + kWalkStages * stage_bytes) + group * (PARTS * 2 * kTiles * 32) + lane;
    const size_t first = (size_t)b.seg_tile0[seg];       // number of the portion's first block
    const uint8_t* recs = p.ws + (first * p.heads + h) * rec_bytes;
    // values: the batch's rows, or those the preparation left (passed through silu), 32 rows per block
    const bool own_v = !kDelta && p.silu;
    const float* vsrc = own_v ? p.v_ws + first * kChunk * p.heads * p.dv + (size_t)h * p.dv + col0 : p.v + (size_t)start * p.ldv + (size_t)h * p.dv + col0;
    const size_t ldv = own_v ? (size_t)p.heads * p.dv : (size_t)p.ldv;
    auto issue = [&](int blk) {
        uint8_t* dst = cw_sm + (blk % kWalkStages) * stage_bytes;
        if (threadIdx.x == 0) {
            constexpr uint32_t skip = kDelta ? 0 : 2 * kPlane;
            const uint8_t* src = recs + (size_t)blk * p.heads * rec_bytes;
            mb_expect(landed + blk % kWalkStages, rec_bytes - skip);
            tma_g2s(dst + skip, src + skip, rec_bytes - skip, landed + blk % kWalkStages);
        }
        float* dv = reinterpret_cast<float*>(dst + rec_bytes);
        const int n = min(kChunk, len - blk * kChunk);
        const float* vb = vsrc + (size_t)blk * kChunk * ldv;
        if (vec) {
            for (int i = threadIdx.x; i < kChunk * kCols / 4; i += kThreads) {
                const int tok = i / (kCols / 4), j = (i % (kCols / 4)) * 4;
                const bool has = tok < n && col0 + j < p.dv;
                cp_async16(dv + tok * kCols + j, has ? vb + tok * ldv + j : vsrc, has ? 16 : 0);
            }
        } else {
            for (int i = threadIdx.x; i < kChunk * kCols; i += kThreads) {
                const int tok = i / kCols, j = i % kCols;
                const bool has = tok < n && col0 + j < p.dv;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dv + i)), "l"(has ? vb + tok * ldv + j : p.v), "r"(has ? 4 : 0) : "memory");
            }
        }
        cp_async_commit();
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < kWalkStages; ++i) mb_init(landed + i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (blocks > 0) issue(0);
    if (blocks > 1) issue(1);
    else cp_async_commit();
    float* st = p.state + ((size_t)slot * p.heads + h) * p.dk * p.dv;
    float S[2 * HS][4];                                  // S^T: rows r0 / r1, columns (key channels) k0 * 16 + nt * 8 + 2c, + 1
#pragma unroll
    for (int nt = 0; nt < 2 * HS; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int ch = k0 * 16 + nt * 8 + 2 * c + (e & 1);
            S[nt][e] = (e < 2 ? ok0 : ok1) && ch < p.dk ? st[(size_t)ch * p.dv + (e < 2 ? r0 : r1)] : 0.0f;
        }
    const bool work = col0 + group * 16 < p.dv;          // the same answer in all warps of a group
    float* orow = p.o + (size_t)(start + 2 * c) * p.ldo + (size_t)h * p.dv + r0;
    for (int blk = 0; blk < blocks; ++blk, orow += (size_t)kChunk * p.ldo) {
        cp_async_wait<1>();
        mb_wait(landed + blk % kWalkStages, (uint32_t)(blk / kWalkStages) & 1);
        __syncthreads();                                 // this block has landed for everyone, and everyone has left the block before
        if (blk + 2 < blocks) issue(blk + 2);
        else cp_async_commit();
        if (!work) continue;
        const uint8_t* rec = cw_sm + (blk % kWalkStages) * stage_bytes;
        const uint4* Kh = reinterpret_cast<const uint4*>(rec) + k0 * 32 + lane;                 // second half of the tokens: KS * 32 pieces further
        const uint4* Kl = Kh + kPlane / 16;
        const uint4* Qh = Kl + kPlane / 16;
        const uint4* Ql = Qh + kPlane / 16;
        const uint4* Eh = Ql + kPlane / 16;              // keys decayed to the block's end
        const uint4* El = Eh + kPlane / 16;
        const uint4* Mh = reinterpret_cast<const uint4*>(rec + 6 * kPlane) + lane;              // M hi, M lo, B hi, B lo: three blocks of 32 pieces each
        const float* D = reinterpret_cast<const float*>(rec + 6 * kPlane + 12 * 512) + k0 * 16 + 2 * c;
        const float* sv = reinterpret_cast<const float*>(rec + rec_bytes) + 2 * c * kCols + cl;
        float x[kTiles][4] = {}, xl[kTiles][4] = {}, xm[kTiles][4] = {}, o[kTiles][4] = {}, ol[kTiles][4] = {}, om[kTiles][4] = {};     // rows r0 / r1, columns (tokens) nt * 8 + 2c, + 1
#pragma unroll
        for (int ks = 0; ks < HS; ++ks) {
            uint32_t ah[4], al[4];
            split_bf16(S[2 * ks][0], S[2 * ks][1], &ah[0], &al[0]);
            split_bf16(S[2 * ks][2], S[2 * ks][3], &ah[1], &al[1]);
            split_bf16(S[2 * ks + 1][0], S[2 * ks + 1][1], &ah[2], &al[2]);
            split_bf16(S[2 * ks + 1][2], S[2 * ks + 1][3], &ah[3], &al[3]);
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                if (kDelta) {
                    const uint4 kh = Kh[(pr * KS + ks) * 32], kl = Kl[(pr * KS + ks) * 32];
                    mma_split<false>(x[2 * pr], xl[2 * pr], xm[2 * pr], ah, al, kh.x, kh.y, kl.x, kl.y);
                    mma_split<false>(x[2 * pr + 1], xl[2 * pr + 1], xm[2 * pr + 1], ah, al, kh.z, kh.w, kl.z, kl.w);
                }
                const uint4 qh = Qh[(pr * KS + ks) * 32], ql = Ql[(pr * KS + ks) * 32];
                mma_split<false>(o[2 * pr], ol[2 * pr], om[2 * pr], ah, al, qh.x, qh.y, ql.x, ql.y);
                mma_split<false>(o[2 * pr + 1], ol[2 * pr + 1], om[2 * pr + 1], ah, al, qh.z, qh.w, ql.z, ql.w);
            }
        }
        auto sum3 = [](const float (&p0)[4], const float (&p1)[4], const float (&p2)[4]) {
            return make_float4(p0[0] + (p1[0] + p2[0]), p0[1] + (p1[1] + p2[1]), p0[2] + (p1[2] + p2[2]), p0[3] + (p1[3] + p2[3]));
        };
        float4* mine = exchange + part * 2 * kTiles * 32;
#pragma unroll
        for (int nt = 0; nt < kTiles; ++nt) {
            if (kDelta) mine[nt * 32] = sum3(x[nt], xl[nt], xm[nt]);
            mine[(kTiles + nt) * 32] = sum3(o[nt], ol[nt], om[nt]);
        }
#pragma unroll
        for (int nt = 0; nt < 2 * HS; ++nt) {            // the old state decays to the block's end
            const float2 d = *reinterpret_cast<const float2*>(D + nt * 8);
            S[nt][0] *= d.x;
            S[nt][1] *= d.y;
            S[nt][2] *= d.x;
            S[nt][3] *= d.y;
        }
        float v[kTiles][4];
#pragma unroll
        for (int nt = 0; nt < kTiles; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) v[nt][e] = sv[(nt * 8 + (e & 1)) * kCols + (e < 2 ? 0 : 8)];
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(PARTS * 32) : "memory");   // the warps of the group
        if (kDelta) {
#pragma unroll
            for (int nt = 0; nt < kTiles; ++nt) {
                float4 y = exchange[nt * 32];
#pragma unroll
                for (int q = 1; q < PARTS; ++q) {
                    const float4 z = exchange[(q * 2 * kTiles + nt) * 32];
                    y = make_float4(y.x + z.x, y.y + z.y, y.z + z.z, y.w + z.w);
                }
                v[nt][0] -= y.x;
                v[nt][1] -= y.y;
                v[nt][2] -= y.z;
                v[nt][3] -= y.w;
            }
        }
        uint32_t uh[2][4], ul[2][4], u3[2][4];
        auto operand = [&](const float (&y)[kTiles][4]) {     // rows x 2 times 16 tokens as A fragments
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                split_bf16(y[2 * pr][0], y[2 * pr][1], &uh[pr][0], &ul[pr][0]);
                split_bf16(y[2 * pr][2], y[2 * pr][3], &uh[pr][1], &ul[pr][1]);
                split_bf16(y[2 * pr + 1][0], y[2 * pr + 1][1], &uh[pr][2], &ul[pr][2]);
                split_bf16(y[2 * pr + 1][2], y[2 * pr + 1][3], &uh[pr][3], &ul[pr][3]);
            }
        };
        operand(v);
        if (kDelta) {
            float u[kTiles][4] = {}, lo[kTiles][4] = {}, mid[kTiles][4] = {};
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    const uint4 mh = Mh[(i + j) * 32], ml = Mh[(3 + i + j) * 32];
                    mma_split<true>(u[2 * i], lo[2 * i], mid[2 * i], uh[j], ul[j], mh.x, mh.y, ml.x, ml.y);
                    mma_split<true>(u[2 * i + 1], lo[2 * i + 1], mid[2 * i + 1], uh[j], ul[j], mh.z, mh.w, ml.z, ml.w);
                }
#pragma unroll
            for (int nt = 0; nt < kTiles; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) u[nt][e] += lo[nt][e] + mid[nt][e];
            operand(u);
            if (kThird) {
                auto rest = [](float a, float b) {
                    uint32_t t1, t2, t3;
                    split3_bf16(a, b, t1, t2, t3);
                    return t3;
                };
#pragma unroll
                for (int pr = 0; pr < 2; ++pr) {
                    u3[pr][0] = rest(u[2 * pr][0], u[2 * pr][1]);
                    u3[pr][1] = rest(u[2 * pr][2], u[2 * pr][3]);
                    u3[pr][2] = rest(u[2 * pr + 1][0], u[2 * pr + 1][1]);
                    u3[pr][3] = rest(u[2 * pr + 1][2], u[2 * pr + 1][3]);
                }
            }
        }
        float add[2 * HS][4] = {};                       // the products of second terms, in accumulators of their own: half as long a chain
#pragma unroll
        for (int pr = 0; pr < 2; ++pr)
#pragma unroll
            for (int ks = 0; ks < HS; ++ks) {
                const uint4 eh = Eh[(pr * KS + ks) * 32], el = El[(pr * KS + ks) * 32];
                mma_bf16_16816(S[2 * ks], uh[pr], eh.x, eh.y);
                mma_bf16_16816(S[2 * ks + 1], uh[pr], eh.z, eh.w);
                mma_bf16_16816(add[2 * ks], ul[pr], eh.x, eh.y);
                mma_bf16_16816(add[2 * ks + 1], ul[pr], eh.z, eh.w);
                mma_bf16_16816(add[2 * ks], uh[pr], el.x, el.y);
                mma_bf16_16816(add[2 * ks + 1], uh[pr], el.z, el.w);
                mma_bf16_16816(add[2 * ks], ul[pr], el.x, el.y);
                mma_bf16_16816(add[2 * ks + 1], ul[pr], el.z, el.w);
                if (kThird) {
                    mma_bf16_16816(add[2 * ks], u3[pr], eh.x, eh.y);
                    mma_bf16_16816(add[2 * ks + 1], u3[pr], eh.z, eh.w);
                }
            }
        // the outputs this warp finishes: tokens mt * 8 + 2c and + 1 of columns r0 and r1
        const int n = min(kChunk, len - blk * kChunk);
#pragma unroll
        for (int m = 0; m < kTiles / PARTS; ++m) {
            const int mt = m * PARTS + part, tok = mt * 8 + 2 * c, i = mt >> 1;
            float y[4] = {}, yl[4] = {}, ym[4] = {};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (j > i) continue;
                const uint4 bh = Mh[(6 + i + j) * 32], bl = Mh[(9 + i + j) * 32];
                if (mt & 1) mma_split<true>(y, yl, ym, uh[j], ul[j], bh.z, bh.w, bl.z, bl.w);
                else mma_split<true>(y, yl, ym, uh[j], ul[j], bh.x, bh.y, bl.x, bl.y);
                if (kThird) mma_bf16_16816(ym, u3[j], mt & 1 ? bh.z : bh.x, mt & 1 ? bh.w : bh.y);
            }
            float4 z = exchange[(kTiles + mt) * 32];
#pragma unroll
            for (int q = 1; q < PARTS; ++q) {
                const float4 w = exchange[(q * 2 * kTiles + kTiles + mt) * 32];
                z = make_float4(z.x + w.x, z.y + w.y, z.z + w.z, z.w + w.w);
            }
            float* to = orow + (size_t)(mt * 8) * p.ldo;
            if (ok0 && tok < n) to[0] = y[0] + (yl[0] + ym[0]) + z.x;
            if (ok0 && tok + 1 < n) to[p.ldo] = y[1] + (yl[1] + ym[1]) + z.y;
            if (ok1 && tok < n) to[8] = y[2] + (yl[2] + ym[2]) + z.z;
            if (ok1 && tok + 1 < n) to[p.ldo + 8] = y[3] + (yl[3] + ym[3]) + z.w;
        }
#pragma unroll
        for (int nt = 0; nt < 2 * HS; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[nt][e] += add[nt][e];
    }
#pragma unroll
    for (int nt = 0; nt < 2 * HS; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int ch = k0 * 16 + nt * 8 + 2 * c + (e & 1);
            if ((e < 2 ? ok0 : ok1) && ch < p.dk) st[(size_t)ch * p.dv + (e < 2 ? r0 : r1)] = S[nt][e];
        }
}

template <int KS, int PARTS, int GROUPS, bool kDelta>
static int launch_walk(const ChunkArgs& p, int vec, cudaStream_t st) {
    constexpr size_t smem = kWalkStages * (chunk_record_bytes(KS * 16) + kChunk * GROUPS * 16 * 4) + GROUPS * PARTS * 2 * (kChunk / 8) * 32 * sizeof(float4);
    SLLM_CUDA(cudaFuncSetAttribute(seq_chunk_walk_kernel<KS, PARTS, GROUPS, kDelta>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    seq_chunk_walk_kernel<KS, PARTS, GROUPS, kDelta><<<dim3(p.b.nseg, p.heads, (p.dv + GROUPS * 16 - 1) / (GROUPS * 16)), PARTS * GROUPS * 32, smem, st>>>(p, vec);
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}

template <int kMode, int dkp>
static int launch_prepare_as(const ChunkArgs& p, int vec, cudaStream_t st) {
    constexpr int smem = ChunkPrepShared<kMode, dkp>::kBytes;
    SLLM_CUDA(cudaFuncSetAttribute(seq_chunk_prepare_kernel<kMode, dkp>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    seq_chunk_prepare_kernel<kMode, dkp><<<dim3(p.b.n_qtiles, p.heads), kPrepThreads, smem, st>>>(p, vec);
    ++g_launches;
    SLLM_LAUNCH_CHECK();
    return SLLM_OK;
}
template <int kMode>
static int launch_prepare(const ChunkArgs& p, int vec, cudaStream_t st) {
    const int dkp = chunk_key(p.dk);
    return dkp == 32 ? launch_prepare_as<kMode, 32>(p, vec, st) : dkp == 64 ? launch_prepare_as<kMode, 64>(p, vec, st) : dkp == 96 ? launch_prepare_as<kMode, 96>(p, vec, st)
                                                                                                                                : launch_prepare_as<kMode, 128>(p, vec, st);
}

template <bool kDelta>
static int launch_chunk_as(ChunkArgs p, cudaStream_t st) {
    const int dkp = chunk_key(p.dk);
    p.v_ws = reinterpret_cast<float*>(p.ws + (size_t)p.b.n_qtiles * p.heads * chunk_record_bytes(dkp));
    auto aligned = [](const void* q) { return ((uintptr_t)q % 16) == 0; };
    const int vec_prep = p.dk % 4 == 0 && p.dv % 4 == 0 && p.ldq % 4 == 0 && p.ldk % 4 == 0 && p.ldv % 4 == 0 && aligned(p.q) && aligned(p.k) && aligned(p.v) &&
                         (!p.channel || (p.lda % 4 == 0 && aligned(p.al) && aligned(p.dt_bias)));
    if (int rc = kDelta ? (p.channel ? launch_prepare<kDecayChannel>(p, vec_prep, st) : launch_prepare<kDecayHead>(p, vec_prep, st)) : launch_prepare<kDecayConstant>(p, vec_prep, st)) return rc;
    const bool own_v = !kDelta && p.silu;
    const int vec = p.dv % 4 == 0 && (own_v || (p.ldv % 4 == 0 && ((uintptr_t)p.v % 16) == 0));
    // a walk is a chain of dependent blocks: few heads are spread over the machine 16 value columns a CTA, many take 32 (every CTA of a head
    // loads all of the head's records)
    const bool narrow = (long long)p.b.nseg * p.heads * ((p.dv + 31) / 32) < sm_count() / 2;
    if (dkp == 32) return narrow ? launch_walk<2, 2, 1, kDelta>(p, vec, st) : launch_walk<2, 2, 2, kDelta>(p, vec, st);
    if (dkp == 64) return narrow ? launch_walk<4, 4, 1, kDelta>(p, vec, st) : launch_walk<4, 4, 2, kDelta>(p, vec, st);
    if (dkp == 96) return narrow ? launch_walk<6, 2, 1, kDelta>(p, vec, st) : launch_walk<6, 2, 2, kDelta>(p, vec, st);
    return narrow ? launch_walk<8, 4, 1, kDelta>(p, vec, st) : launch_walk<8, 4, 2, kDelta>(p, vec, st);
}

// Whether a step goes in blocks of 16 tokens. The lengths of the portions are on the device: their mean stands for them. Measured, us, both kernels, 16 | 32 tokens a block.
// - Many CTAs (a portion, head and 32 value columns each): those of blocks of 32 fill an SM alone (128 key channels) or in pairs. Heads of 128, 16 of them: 8 portions of 64, 128 and 300 43 | 41, 78 | 73,
//   166 | 160, 32 portions of 16, 40 and 100 53 | 79, 111 | 138, 232 | 250; 8 heads of 64: 8 portions of 100 23 | 21, 32 portions of 40 and 100 33 | 39, 63 | 69; 8 heads of 32: 32 of 40 20 | 21.
// - Portions that end in the first half of a block: one of 33 tokens 14 | 15, of 64 15 | 15, of 80 16 | 17, of 128 20 | 19, of 300 37 | 31; 8 of 40 37 | 40, of 50 42 | 40, of 70 52 | 54.
// - A constant decay needs no triangle inverted, so the larger blocks' matrices weigh more (heads of 128): one of 64 12 | 14, of 128 15 | 16, of 160 18 | 17, of 2048 142 | 112; two of 64 14 | 16, of 150 22 | 22; 8
//   of 100 and 300 47 | 54, 113 | 120.
// - A decay per channel takes an exponential per channel and pair of rows: 16 heads of 128, one of 300 38 | 41, of 600 65 | 70, of 1000 105 | 100, two of 300 55 | 65, 8 of 100 71 | 94; 8 heads of 64, one of 200 22 | 23, of 300
//   29 | 27, of 1000 74 | 59; 8 heads of 32, one of 200 18 | 19, of 400 28 | 26. What a longer chain costs (0.26 us a block of 16) stands against the work per block and head.
static bool chunk_in_16(const ChunkArgs& p) {
    const int dkp = chunk_key(p.dk);
    const long long T = p.b.T, nseg = p.b.nseg, ctas = nseg * p.heads * ((p.dv + 31) / 32);
    if (p.delta && p.channel) return nseg > 1 || T * (44 - (dkp > 64 ? 2 : 1) * p.heads) <= 11000;
    if (!p.delta) return ctas > sm_count() || T < 140 * nseg;
    if (ctas > (dkp > 96 ? 4LL : dkp > 64 ? 3LL : dkp > 32 ? 2LL : 1LL) * sm_count()) return true;
    return T <= 90 * nseg && ((T + 16 * nseg - 1) / (16 * nseg)) % 2 == 1;
}

int launch_chunk_scan(const ChunkArgs& p, cudaStream_t st) {
    SLLM_REQUIRE(p.dk <= kChunkMaxKey && p.ws && ((uintptr_t)p.ws % 16) == 0 && p.b.seg_tile0 && p.b.qt_seg && p.b.qt_off && p.b.n_qtiles > 0, SLLM_EINVAL,
                 "chunk scan: heads of %d key channels, or an incomplete batch description", p.dk);
    if (chunk_in_16(p)) return launch_chunk16_scan(p, st);
    return p.delta ? launch_chunk_as<true>(p, st) : launch_chunk_as<false>(p, st);
}

}  // namespace sllm

extern "C" int64_t sllm_seq_chunk_ws_bytes(int32_t n_qtiles, int32_t heads, int32_t dk, int32_t dv) {
    return dk > 0 && dk <= sllm::kChunkMaxKey && dv > 0 && n_qtiles > 0 && heads > 0 ? (int64_t)sllm::chunk_ws_bytes(n_qtiles, heads, dk, dv) : 0;
}
