// csrc/mega_common.cuh — device helpers shared by the two persistent decode-step kernels
// (megakernel.cu: grid-barrier version; megakernel_ll.cu: barrier-free {value, epoch}-word version).
#pragma once
#include "megakernel.cuh"

namespace sllm {

constexpr int kMegaThreads = 512;
constexpr int kMegaWarps = kMegaThreads / 32;
constexpr int kSlotBytes = 4096;
static_assert(kSlotBytes == kTileSlotBytes, "tile geometry and ring slot size must agree");
constexpr int kSlots = 2;
constexpr int kCplMax = 4;        // max 16-byte chunks per lane per row slice (slice <= 2 KB)
constexpr int kRoundUnits = 128;  // units per partial-table round
constexpr int kAttTile = 64;
constexpr int kAttP = 3 * kAttTile;   // scores per query head the single-pass attention of megakernel2.cu keeps (two K/V stages + a tail of <= 64 rows)
constexpr unsigned kSpinLimit = 1u << 26;
#ifndef SLLM_BARRIER_POLL_COUNTER
#define SLLM_BARRIER_POLL_COUNTER 1   // measured on B200 (llama2-7b bf16): 350.4 tok/s vs 338.1 with the separate release flag
#endif
constexpr int kAttRecPad = 4;     // partial record = hd floats of O, then m, l (+2 pad: keeps float4 alignment)


struct MegaSmem {
    size_t bars, red, part, ring, att, total;
    size_t att_q, att_p, att_misc, att_k, att_v;
    int kv_stride;
    int att_tile;   // cache positions per K/V stage: 64, or 32 when a row is wider than 256 bytes (fp32 cache with 128-wide heads), so that
                    // two K and two V stages always fit in 64 KB next to the weight rings
};
__host__ __device__ constexpr int mega_att_tile(int hd, int kv_esz) { return hd * kv_esz > 256 ? kAttTile / 2 : kAttTile; }
__host__ __device__ inline int mega_kv_stride(int row_bytes) {
    int s = (row_bytes / 128) * 128 + 32;
    if (s < row_bytes) s += 128;
    return s;
}
__host__ __device__ constexpr MegaSmem mega_smem_layout(int hd, int g, int kv_esz) {
    MegaSmem L{};
    size_t off = 0;
    L.bars = off; off += 512;
    L.red = off; off += 256;
    L.part = off; off += (size_t)kRoundUnits * 2 * kMegaWarps * 4;
    off = (off + 127) & ~(size_t)127;
    L.ring = off; off += (size_t)kMegaWarps * kSlots * kSlotBytes;
    L.att = off;
    L.att_q = off; off += (size_t)g * hd * 4;
    L.att_p = off; off += (size_t)g * kAttP * 4;
    L.att_misc = off; off += 256;
    off = (off + 127) & ~(size_t)127;
    L.kv_stride = hd * kv_esz;   // dense rows: a tile is one contiguous bulk copy
    L.att_tile = mega_att_tile(hd, kv_esz);
    L.att_k = off; off += (size_t)2 * L.att_tile * L.kv_stride;
    L.att_v = off; off += (size_t)2 * L.att_tile * L.kv_stride;
    L.total = off;
    return L;
}

// ------------------------------------------------------------------------------------- primitives ----
__device__ __forceinline__ uint32_t s_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mb_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mb_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mb_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    unsigned spins = 0;
    do {
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(s_addr(bar)), "r"(parity) : "memory");
        if (!done && ++spins > kSpinLimit) __trap();
    } while (!done);
}
__device__ __forceinline__ void tma_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(s_addr(dst)), "l"(src), "r"(bytes), "r"(s_addr(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// grid-wide barrier (cooperative launch guarantees co-residency). counter[0] = arrivals (monotonic across launches; wrap-safe
// compares). Default: thread 0 of every CTA arrives with ONE atom.add.release and then polls the counter itself with ld.acquire
// until the target — the last arriver needs no extra hop to publish anything (measured: 2.85 ms/token instead of 2.96 with the
// older scheme, kept under SLLM_BARRIER_POLL_COUNTER=0: fence + atomicAdd, the last arriver stores the epoch to counter[32] on
// its own 128-byte line, the others poll that line; relaxed polls + one acquire fence were slower (346 tok/s), a 40 ns back-off
// between polls made no difference). No trailing fence: every cross-CTA read in this kernel is an L2 access
// (ld.global.cg or TMA), never an L1-cached load.
__device__ __forceinline__ void grid_barrier(unsigned* counter, unsigned target) {
    __syncthreads();
    if (threadIdx.x == 0) {
#if SLLM_BARRIER_POLL_COUNTER
        unsigned v;
        asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(counter) : "memory");
        v += 1u;
        unsigned spins = 0;
        while ((int)(v - target) < 0) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if (++spins > kSpinLimit) __trap();
        }
#else
        __threadfence();
        const unsigned prev = atomicAdd(counter, 1u);
        if (prev + 1u == target) {
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(counter + 32), "r"(target) : "memory");
        } else {
            unsigned spins = 0;
            while (true) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter + 32) : "memory");
                if ((int)(v - target) >= 0) break;
                if (++spins > kSpinLimit) __trap();
            }
        }
#endif
    }
    __syncthreads();
}

__device__ __forceinline__ void unit_rows(const MegaParams& p, const PhaseDesc& ph, int u, int& r0, int& r1) {
    if (ph.kind == PH_QKV) {
        const int half = p.hd >> 1, rope_units = (p.q_loc + p.kv_loc) >> 1;
        if (u < rope_units) {
            const int head = u / half, j = u - head * half;
            r0 = head * p.hd + j;
            r1 = r0 + half;
        } else {
            r0 = p.q_loc + p.kv_loc + 2 * (u - rope_units);
            r1 = r0 + 1;
        }
    } else if (ph.kind == PH_GATEUP) {
        r0 = u;
        r1 = p.I_loc + u;
    } else {
        r0 = 2 * u;
        r1 = min(2 * u + 1, ph.nrows - 1);
    }
}

// balanced split of a phase's tile rows over the CTAs
__device__ __forceinline__ int cta_cut(const uint32_t* cum, int n, int cta, int ncta) {   // first of CTA `cta`'s share of n items
    return cum ? (int)(((uint64_t)n * cum[cta]) >> 24) : (int)(((int64_t)n * cta) / ncta);
}
__device__ __forceinline__ void cta_tiles(const PhaseDesc& ph, int cta, int ncta, int& g0, int& g1) {
    g0 = cta_cut(ph.cum, ph.ntr, cta, ncta);
    g1 = cta_cut(ph.cum, ph.ntr, cta + 1, ncta);
}

// the split a phase's tile rows get in the kernel that fuses the down projection into the gate_up phase: gate_up follows the split
// of the (transposed) down matrix, whose tile rows are kFuseJT units, so that a CTA multiplies exactly the values it produced
template <bool FUSE>
__device__ __forceinline__ void phase_tiles(const PhaseDesc& ph, int cta, int ncta, int& g0, int& g1) {
    if (FUSE && ph.kind == PH_GATEUP) {
        const int per = kFuseJT / (ph.R >> 1);        // gate_up tile rows (R / 2 units each) per down tile row
        const int ntr_e = ph.nunits / kFuseJT;
        g0 = cta_cut(ph.cum, ntr_e, cta, ncta) * per;
        g1 = cta_cut(ph.cum, ntr_e, cta + 1, ncta) * per;
    } else {
        cta_tiles(ph, cta, ncta, g0, g1);
    }
}

// The CTA's share of a phase ([first, last) tile rows; for PH_WO_T of its item), worked out once per launch and kept where the descriptor's table pointer was: from
// the table, an L2 round trip, or by 64-bit divisions it stood on the path of every producer that came to a new phase, as good as every tile of a small model.
__device__ __forceinline__ const uint32_t* pack_share(int first, int last) {
    return reinterpret_cast<const uint32_t*>((uint64_t)(uint32_t)first | ((uint64_t)(uint32_t)last << 32));
}
__device__ __forceinline__ void share_of(const PhaseDesc& ph, int& first, int& last) {
    const uint64_t v = reinterpret_cast<uint64_t>(ph.cum);
    first = (int)(uint32_t)v;
    last = (int)(uint32_t)(v >> 32);
}
template <bool FUSE>
__device__ __forceinline__ void keep_share(PhaseDesc& ph, int cta, int ncta, int nsplit) {
    int first, last;
    if (ph.kind == PH_WO_T) {
        const int part = cta % nsplit;
        first = (int)(((int64_t)ph.ntr * part) / nsplit);
        last = (int)(((int64_t)ph.ntr * (part + 1)) / nsplit);
    } else {
        phase_tiles<FUSE>(ph, cta, ncta, first, last);
    }
    ph.cum = pack_share(first, last);
}

// tile rows [a, b) of the transposed down matrix that row group rg of RG takes out of a CTA's [g0, g1): contiguous shares
__device__ __forceinline__ void down_t_rows(int g0, int g1, int rg, int RG, int& a, int& b) {
    const int cnt = g1 - g0;
    a = g0 + (cnt * rg) / RG;
    b = g0 + (cnt * (rg + 1)) / RG;
}

// Attention output of `heads` heads from h0 on, their splits' partial records merged, into xs. A warp turns the maxima and sums of a head's splits into weights, a lane per
// split (a plan has at most 32); then a thread takes every ngrp-th split of one 16-byte piece, eight loads on their way. Bound: round trips to L2. Measured, us a step at
// position 200: 22 layers of TinyLlama's shape (32 heads over 4 kv heads in 32 splits), int8, 1170 with two dependent loops over the splits in every thread, 1278 with all
// of a head's maxima, exponentials and loads one behind the other in every thread, 1115 like this; stories110M (12 heads in 12 splits), fp32, 395, 336 and 326. Pieces asked
// for in front of the weights cost more than the trip they save, since they live through that loop in registers the kernel does not have: eight 1240, four 1160.
// wgt: the partial table, idle here; xs_bytes: what lies behind xs.
__device__ __forceinline__ void merge_splits(const MegaParams& p, int h0, int heads, float* xs, size_t xs_bytes, float* wgt) {
    constexpr int kAhead = 8, kHeads = 4;
    const int tid = threadIdx.x, lane = tid & 31, rec = p.hd + kAttRecPad, ns = p.nsplit, width = heads * p.hd, nc = width / 4;
    const float* base = p.att_part + (size_t)h0 * ns * rec;
    const int ngrp = max(1, min(min(kMegaThreads / nc, ns), (int)(xs_bytes / ((size_t)width * 4)) - 1));
    const int grp = ngrp > 1 ? tid / nc : 0, per = ngrp > 1 ? nc : kMegaThreads;
    float* share = xs + width;                  // [ngrp][nc] pieces
    float* sums = wgt + heads * ns;             // [heads], behind the weights [heads][ns]
    const int c0 = tid - grp * nc;
    const bool takes = grp < ngrp && c0 < nc;
    float4 v[kAhead];
    auto ask = [&](int c4, int s0) {
        const int h = c4 * 4 / p.hd;
        const float* src = base + (size_t)h * ns * rec + (c4 * 4 - h * p.hd);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s0 + k * ngrp < ns) v[k] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(s0 + k * ngrp) * rec));
        }
    };
    for (int first = tid >> 5; first < heads; first += kHeads * kMegaWarps) {
        float m[kHeads], l[kHeads];
#pragma unroll
        for (int k = 0; k < kHeads; ++k) {
            const int h = first + k * kMegaWarps;
            m[k] = -INFINITY;
            l[k] = 0.f;
            if (h < heads && lane < ns) {
                const float* r = base + ((size_t)h * ns + lane) * rec + p.hd;
                m[k] = __ldcg(r);
                l[k] = __ldcg(r + 1);
            }
        }
#pragma unroll
        for (int k = 0; k < kHeads; ++k) {
            const int h = first + k * kMegaWarps;
            if (h >= heads) break;
            const float M = warp_max(m[k]), w = m[k] == -INFINITY ? 0.f : expf(m[k] - M), sum = warp_sum(l[k] * w);
            if (lane < ns) wgt[h * ns + lane] = w;
            if (lane == 0) sums[h] = sum;
        }
    }
    __syncthreads();
    if (takes) {
        for (int c4 = c0; c4 < nc; c4 += per) {
            const int h = c4 * 4 / p.hd;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int s0 = grp; s0 < ns; s0 += kAhead * ngrp) {
                ask(c4, s0);
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    const float w = s0 + k * ngrp < ns ? wgt[h * ns + s0 + k * ngrp] : 0.f;
                    o.x = fmaf(v[k].x, w, o.x); o.y = fmaf(v[k].y, w, o.y); o.z = fmaf(v[k].z, w, o.z); o.w = fmaf(v[k].w, w, o.w);
                }
            }
            if (ngrp == 1) {
                const float Ls = sums[h];
                reinterpret_cast<float4*>(xs)[c4] = make_float4(o.x / Ls, o.y / Ls, o.z / Ls, o.w / Ls);
            } else {
                reinterpret_cast<float4*>(share)[grp * nc + c4] = o;
            }
        }
    }
    if (ngrp == 1) return;                      // callers synchronise
    __syncthreads();
    if (tid < nc) {
        float4 o = reinterpret_cast<const float4*>(share)[tid];
        for (int g = 1; g < ngrp; ++g) {
            const float4 q = reinterpret_cast<const float4*>(share)[g * nc + tid];
            o.x += q.x; o.y += q.y; o.z += q.z; o.w += q.w;
        }
        const float Ls = sums[tid * 4 / p.hd];
        reinterpret_cast<float4*>(xs)[tid] = make_float4(o.x / Ls, o.y / Ls, o.z / Ls, o.w / Ls);
    }
}

// Norm weights of this layer's second half and of the next layer, asked into L2 while it is early: a phase needs them right behind a barrier.
__device__ __forceinline__ void prefetch_norms(const MegaParams& p, int l, int cta, int ncta) {
    const int lines = (p.d * 8 + 127) / 128;
    for (int i = cta + threadIdx.x * ncta; i < lines; i += ncta * kMegaThreads)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t*>(p.norms + (size_t)(2 * l + 1) * p.d) + min(i * 128, p.d * 8 - 4)));
}

// ---- L2 prefetch of the weight stream: built twice, measured, removed ------------------------------------------------------
// The rings hold 128 KB per SM; at a dependency point (grid barrier, attention, per-head counters) the consumers stall and HBM runs dry
// (with the dot products removed the step takes exactly as long, with the barriers removed it is 20 % shorter: r02_mega_debug_v1.jsonl).
// Asking the L2 for the tiles beyond the ring with cp.async.bulk.prefetch.L2 works IN ISOLATION (39 MB asked
// for, 10 us of idling, then streamed through the rings in 2.1 us instead of 4.2 us = 120-130 GB/s per SM against 49-63 from HBM), and
// loses in the kernel in both forms tried: (1) a continuous look-ahead of 2-16 tiles per warp during streaming: -5 % to -30 %; (2) 2-12 tiles per warp asked for right before a grid barrier and / or before the attention chain:
// -4 % to -13 %. A CTA's "stall" is the time the slowest CTAs still stream (the bulk prefetches
// of the early ones take HBM bandwidth from exactly the copies the barrier is waiting for), and the attention / counter chain is a
// sequence of small latency-critical L2 round trips that queue behind 40 MB of prefetch traffic. HBM is the shared resource: anything
// that is not on the critical path and uses it lengthens the critical path.

// acc[e] += w_e * s for the E weights of one 16-byte chunk (fp32 / bf16 storage)
template <int WD>
__device__ __forceinline__ void axpy_chunk(const uint4 w, float s, float* acc) {
    if (WD == SLLM_F32) {
        acc[0] = fmaf(__uint_as_float(w.x), s, acc[0]); acc[1] = fmaf(__uint_as_float(w.y), s, acc[1]);
        acc[2] = fmaf(__uint_as_float(w.z), s, acc[2]); acc[3] = fmaf(__uint_as_float(w.w), s, acc[3]);
    } else {
        acc[0] = fmaf(bf16_lo(w.x), s, acc[0]); acc[1] = fmaf(bf16_hi(w.x), s, acc[1]);
        acc[2] = fmaf(bf16_lo(w.y), s, acc[2]); acc[3] = fmaf(bf16_hi(w.y), s, acc[3]);
        acc[4] = fmaf(bf16_lo(w.z), s, acc[4]); acc[5] = fmaf(bf16_hi(w.z), s, acc[5]);
        acc[6] = fmaf(bf16_lo(w.w), s, acc[6]); acc[7] = fmaf(bf16_hi(w.w), s, acc[7]);
    }
}
__device__ __forceinline__ void red_add_v4(float* dst, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <int KVD> struct MKv;
template <> struct MKv<SLLM_F32> { static constexpr int ESZ = 4, VEC = 4; };
template <> struct MKv<SLLM_BF16> { static constexpr int ESZ = 2, VEC = 8; };

template <int KVD>
__device__ __forceinline__ void kv_unpack(const uint4 v, float* f) {
    if (KVD == SLLM_F32) {
        f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
    } else {
        f[0] = bf16_lo(v.x); f[1] = bf16_hi(v.x); f[2] = bf16_lo(v.y); f[3] = bf16_hi(v.y);
        f[4] = bf16_lo(v.z); f[5] = bf16_hi(v.z); f[6] = bf16_lo(v.w); f[7] = bf16_hi(v.w);
    }
}

// 16 bytes of weights (E elements) times E activations held in registers
template <int WD>
__device__ __forceinline__ float reg_dot(const uint4 w, const float* x, float acc) {
    if (WD == SLLM_F32) {
        acc = fmaf(__uint_as_float(w.x), x[0], acc); acc = fmaf(__uint_as_float(w.y), x[1], acc);
        acc = fmaf(__uint_as_float(w.z), x[2], acc); acc = fmaf(__uint_as_float(w.w), x[3], acc);
    } else if (WD == SLLM_INT8) {   // unscaled: the caller multiplies by the chunk's group scale
        acc = word_dot_s8(w.x, make_float4(x[0], x[1], x[2], x[3]), acc);
        acc = word_dot_s8(w.y, make_float4(x[4], x[5], x[6], x[7]), acc);
        acc = word_dot_s8(w.z, make_float4(x[8], x[9], x[10], x[11]), acc);
        acc = word_dot_s8(w.w, make_float4(x[12], x[13], x[14], x[15]), acc);
    } else {
        acc = fmaf(bf16_lo(w.x), x[0], acc); acc = fmaf(bf16_hi(w.x), x[1], acc);
        acc = fmaf(bf16_lo(w.y), x[2], acc); acc = fmaf(bf16_hi(w.y), x[3], acc);
        acc = fmaf(bf16_lo(w.z), x[4], acc); acc = fmaf(bf16_hi(w.z), x[5], acc);
        acc = fmaf(bf16_lo(w.w), x[6], acc); acc = fmaf(bf16_hi(w.w), x[7], acc);
    }
    return acc;
}


__device__ __forceinline__ void warp_better(float& v, int& i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) better_of(v, i, __shfl_xor_sync(0xffffffffu, v, o), __shfl_xor_sync(0xffffffffu, i, o));
}
// (v, i) of every thread -> the CTA's best in all threads of warp 0; red: 2 * kMegaWarps words of shared memory
__device__ __forceinline__ void cta_better(float& v, int& i, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* ri = reinterpret_cast<int*>(red + kMegaWarps);
    warp_better(v, i);
    if (lane == 0) { red[warp] = v; ri[warp] = i; }
    __syncthreads();
    if (warp == 0) {
        v = lane < kMegaWarps ? red[lane] : -INFINITY;
        i = lane < kMegaWarps ? ri[lane] : 0x7fffffff;
        warp_better(v, i);
    }
}
// Rows [r0, r1) of the logits into pinned host memory. A function of its own: written out in mega_finish it cost kernels that have no register to spare 2 % of a step.
static __device__ __noinline__ void mega_logits_out(const float* from, float* to, int r0, int r1) {
#pragma unroll 1
    for (int r = (r0 & ~3) + 4 * (int)threadIdx.x; r < r1; r += 4 * kMegaThreads) {
        if (r >= r0 && r + 4 <= r1) {
            *reinterpret_cast<float4*>(to + r) = __ldcg(reinterpret_cast<const float4*>(from + r));
        } else {
#pragma unroll 1
            for (int e = max(r, r0); e < min(r + 4, r1); ++e) to[e] = __ldcg(from + e);
        }
    }
}
// End of the classifier phase: every CTA leaves its best logit, the CTA that comes last picks the arg max and advances the step state. True in the one thread that has
// done so (it stores the counters that its kernel keeps). All threads of the last CTA read the candidates: by one thread, a chain of 148 reads of L2, that end took
// several us. A call that wants its logits on the host (p.call.logits, pinned) gets this CTA's rows [r0, r1) from here: read back from the device's copy, 16 bytes a thread,
// so that a warp stores 512 bytes in a row over PCIe, and behind the ticket, so that no fence waits for them to arrive. kLogits = false: no call asks for them. (Over int8 weights, whose
// kernels have no register to spare, the call that is not taken cost a step of a model 2048 wide 226.5 us instead of 223.)
template <bool kLogits>
__device__ __forceinline__ bool mega_finish(const MegaParams& p, float v, int i, float* red, int* s_last, int cta, int ncta, int r0, int r1) {
    cta_better(v, i, red);
    if (threadIdx.x == 0) {
        p.blk_val[cta] = v;
        p.blk_idx[cta] = i;
        __threadfence();
        *s_last = (atomicAdd(&p.st->ticket, 1) == ncta - 1);
        __threadfence();
    }
    __syncthreads();
    if (kLogits && p.call.logits) mega_logits_out(p.logits, p.call.logits, r0, r1);
    if (!*s_last) return false;
    v = -INFINITY;
    i = 0x7fffffff;
    for (int b = threadIdx.x; b < ncta; b += kMegaThreads) better_of(v, i, __ldcg(p.blk_val + b), __ldcg(p.blk_idx + b));
    cta_better(v, i, red);
    if (threadIdx.x != 0) return false;
    if (i == 0x7fffffff) i = 0;
    p.blk_val[ncta] = v;
    p.blk_idx[ncta] = i;
    p.st->ticket = 0;
    if (p.call.token >= 0) { p.st->pos = p.call.pos; p.st->n_prompt = 0; }
    if (p.call.next) *p.call.next = i;
    ClsPolicy<SLLM_F32>::step_feedback(p.st, p.prompt, p.history, i);
    return true;
}
static __device__ __noinline__ void mega_timeout(const char* what) {
    printf("sllm mega: %s timed out (cta %d warp %d)\n", what, (int)blockIdx.x, (int)(threadIdx.x >> 5));
    __trap();
}
__device__ __forceinline__ void mb_wait_fast(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    unsigned spins = 0;
    do {
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(s_addr(bar)), "r"(parity) : "memory");
        if (!done && ++spins > kSpinLimit) mega_timeout("mbarrier");
    } while (!done);
}


}  // namespace sllm
