// csrc/seq_chunk.cuh — the recurrences of seq_delta.cu in blocks of 32 (seq_chunk.cu) or 16 tokens (seq_chunk16.cu) on the tensor cores: arguments, launch and what both forms share.
#pragma once
#include "seq_attn.cuh"
#include "seq_common.cuh"

namespace sllm {

constexpr int kChunk = 32, kChunk16 = 16;          // tokens of a block: a query tile of the batch description, or half of one
constexpr int kChunkMaxKey = 128;   // key channels of a head, at most

struct ChunkArgs {
    sllm_seq_batch b;
    const float *q, *k, *v; int ldq, ldk, ldv;
    int delta;                                           // 1: delta rule; 0: linear attention with a constant decay
    // delta rule: logits of beta [heads] and of the decay's step ([heads], or [heads * dk] with `channel`), A_log [heads], dt_bias like the step
    const float *bl, *al; int ldb, lda; const float *A_log, *dt_bias; int channel;
    // constant decay: [heads] minus the decay's logarithm; (cos, sin) [T][n_freq] that turn q and k (NULL = not); q, k and v pass silu
    const float* rate; const float2* angles; int n_freq, layout, silu;
    int heads, kv_heads, dk, dv;
    float unit_eps, scale;                               // delta rule: q times scale; constant decay: k times scale
    float* state; float* o; int ldo;
    uint8_t* ws;                                         // chunk_ws_bytes: the blocks' records, then
    float* v_ws;                                         // values passed through silu [blocks][tokens of a block][heads * dv] (set by the launch)
};

// key channels rounded up to what the kernel is instantiated for
__host__ __device__ __forceinline__ int chunk_key(int dk) { return dk <= 32 ? 32 : dk <= 64 ? 64 : dk <= 96 ? 96 : 128; }
// per block and head: decayed keys, decayed queries and keys decayed to the block's end as (hi, lo) bf16 fragments, the lower triangles of the two 32 x 32 matrices (three
// blocks of 16 x 16 each) likewise, the block's decay per key channel
__host__ __device__ constexpr size_t chunk_record_bytes(int dkp) { return (size_t)dkp * (6 * kChunk * 2 + 4) + 12 * 16 * 16 * 2; }
// the same of a block of 16 tokens, whose matrices are one block of 16 x 16
__host__ __device__ constexpr size_t chunk16_record_bytes(int dkp) { return (size_t)dkp * (6 * kChunk16 * 2 + 4) + 4 * 16 * 16 * 2; }
// records and values of either form
inline size_t chunk_ws_bytes(int n_qtiles, int heads, int dk, int dv) {
    const size_t records = chunk_record_bytes(chunk_key(dk)), records16 = 2 * chunk16_record_bytes(chunk_key(dk));
    return (size_t)n_qtiles * heads * ((records > records16 ? records : records16) + (size_t)kChunk * dv * sizeof(float));
}
int launch_chunk_scan(const ChunkArgs& p, cudaStream_t st);        // in whichever blocks suit the step
int launch_chunk16_scan(const ChunkArgs& p, cudaStream_t st);

constexpr float kLog2e = 1.4426950408889634f;

// eight values -> 16 bytes of hi terms and 16 bytes of lo terms
__device__ __forceinline__ void chunk_put(uint8_t* hi, uint8_t* lo, int at, const float (&v)[8]) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) split_bf16(v[2 * i], v[2 * i + 1], &h[i], &l[i]);
    reinterpret_cast<uint4*>(hi)[at] = make_uint4(h[0], h[1], h[2], h[3]);
    reinterpret_cast<uint4*>(lo)[at] = make_uint4(l[0], l[1], l[2], l[3]);
}

// Products of two-term operands: (ah + al) (bh + bl), each term's into an accumulator of its own as far as there are three (no product waits for another). The product of the second
// terms, as large as what two terms leave of an operand, is kept where u is an operand (kAll), and left out of the products with the old state.
template <bool kAll>
__device__ __forceinline__ void mma_split(float (&d)[4], float (&dl)[4], float (&dm)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4], uint32_t h0, uint32_t h1, uint32_t l0, uint32_t l1) {
    mma_bf16_16816(d, ah, h0, h1);
    mma_bf16_16816(dl, al, h0, h1);
    mma_bf16_16816(dm, ah, l0, l1);
    if (kAll) mma_bf16_16816(dl, al, l0, l1);
}

}  // namespace sllm
