// csrc/seq_ssd_block.cuh — state-space duality in blocks of 64 tokens (seq_ssd_block.cu): arguments and scratch layout.
#pragma once
#include "seq_common.cuh"

namespace sllm {

constexpr int kSsdBlock = 64;          // tokens of a block = two query tiles of the batch description
constexpr int kSsdMaxState = 128;      // states per channel, at most

struct SsdBlockArgs {
    sllm_seq_batch b;
    const float *x, *B, *C, *step; int ldx, ldb, ldc, lda;
    const float *A_log, *dt_bias, *skip;
    int heads, groups, n_state, dv;
    float* state; float* y; int ldy;
    uint8_t* group_ws;                 // per (block, group): fragments of C and B, products C_i . B_j
    size_t slots; int32_t* status;     // blocks the scratch has room for; where a batch that needs more is reported
    float* head_ws;                    // per (block, head): running sums of the decays' base-2 logarithms [64] and their second terms [64], step sizes [64]
};

// number of a portion's block in the scratch; portions follow each other with room for a last half block
__host__ __device__ __forceinline__ size_t ssd_block_id(int seg_tile0, int seg, int blk) { return (size_t)(seg_tile0 / 2 + seg + blk); }
inline size_t ssd_block_count(int n_qtiles, int nseg) { return (size_t)(n_qtiles / 2 + nseg + 1); }
constexpr size_t ssd_block_group_bytes(int nk) { return (size_t)8 * (nk / 16) * 512 + (size_t)(nk / 8) * 4 * 512 + 20 * 512; }

}  // namespace sllm
