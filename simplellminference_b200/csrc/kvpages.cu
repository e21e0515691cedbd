// csrc/kvpages.cu — sllm_kvpages_*: the exported face of the page bookkeeping (kvpages.cuh). Its own translation unit so that a
// library holding only part of the kernels can carry it; and sllm_seq_step_fill, the index arrays of a ragged step built from the same tables.
#include <algorithm>
#include <exception>
#include <vector>

#include "kvpages.cuh"

using namespace sllm;

extern "C" {

sllm_kvpages* sllm_kvpages_create(int32_t n_pages, int32_t page_len, int32_t max_seqs, int32_t max_pages_per_seq) {
    if (n_pages < 1 || page_len < 1 || max_seqs < 1 || max_pages_per_seq < 1) {
        set_error("kvpages: n_pages=%d page_len=%d max_seqs=%d max_pages_per_seq=%d must all be positive", n_pages, page_len, max_seqs, max_pages_per_seq);
        return nullptr;
    }
    auto* kp = new sllm_kvpages();
    kp->n_pages = n_pages; kp->page_len = page_len; kp->max_seqs = max_seqs; kp->max_pages = max_pages_per_seq;
    kp->free_.resize(n_pages);
    for (int i = 0; i < n_pages; ++i) kp->free_[i] = n_pages - 1 - i;
    kp->table.assign((size_t)max_seqs * max_pages_per_seq, -1);
    kp->held.assign(max_seqs, 0);
    return kp;
}

void sllm_kvpages_destroy(sllm_kvpages* kp) { delete kp; }

int32_t sllm_kvpages_reserve(sllm_kvpages* kp, int32_t seq, int32_t n_positions) {
    SLLM_REQUIRE(kp && seq >= 0 && seq < kp->max_seqs && n_positions >= 0, SLLM_EINVAL, "kvpages_reserve: bad argument (seq %d, positions %d)", seq, n_positions);
    const int extra = kp->extra_needed(seq, n_positions);
    SLLM_REQUIRE(extra >= 0, SLLM_EINVAL, "kvpages_reserve: %d positions need more than %d pages of %d", n_positions, kp->max_pages, kp->page_len);
    SLLM_REQUIRE(extra <= (int)kp->free_.size(), SLLM_ENOMEM, "out of KV pages: sequence %d needs %d more, %d free", seq, extra, (int)kp->free_.size());
    kp->take(seq, extra);
    return extra;
}

int sllm_kvpages_release(sllm_kvpages* kp, int32_t seq) {
    SLLM_REQUIRE(kp && seq >= 0 && seq < kp->max_seqs, SLLM_EINVAL, "kvpages_release: bad sequence %d", seq);
    kp->release(seq);
    return SLLM_OK;
}

int32_t sllm_kvpages_free_count(const sllm_kvpages* kp) { return kp ? (int32_t)kp->free_.size() : 0; }
int32_t sllm_kvpages_held(const sllm_kvpages* kp, int32_t seq) { return (kp && seq >= 0 && seq < kp->max_seqs) ? kp->held[seq] : 0; }
const int32_t* sllm_kvpages_table(const sllm_kvpages* kp) { return kp ? kp->table.data() : nullptr; }

int64_t sllm_seq_step_fill(int32_t* out, int64_t capacity, int32_t nseg, const int32_t* segments, const int32_t* tokens, const int32_t* rows, int32_t n_rows,
                           const sllm_kvpages* kp, int32_t tile, int64_t* offsets, int32_t* n_qtiles) {
    SLLM_REQUIRE(nseg > 0 && segments && tokens && kp && tile > 0 && offsets && n_qtiles && n_rows >= 0 && (n_rows == 0 || rows), SLLM_EINVAL, "seq_step_fill: bad argument");
    if (int rc = status_check()) return rc;          // what an earlier step left unfinished
    int64_t T = 0, tiles = 0;
    for (int i = 0; i < nseg; ++i) {
        const int32_t len = segments[4 * i + 2];
        SLLM_REQUIRE(len > 0 && segments[4 * i + 1] >= 0 && segments[4 * i] >= 0 && segments[4 * i] < kp->max_seqs, SLLM_EINVAL, "seq_step_fill: segment %d", i);
        T += len;
        tiles += (len + tile - 1) / tile;
    }
    const int64_t table = (int64_t)kp->max_seqs * kp->max_pages;
    // ids, token slots, token positions | segment starts, lengths, slots, first positions | tiles' segments, offsets | rows | block table | segments' first tiles | previous ids
    const int64_t sizes[13] = {T, T, T, nseg, nseg, nseg, nseg, tiles, tiles, std::max(1, n_rows), table, nseg, T};
    int64_t total = 0;
    for (int i = 0; i < 13; ++i) {
        offsets[i] = total;
        total += sizes[i];
    }
    *n_qtiles = (int32_t)tiles;
    if (!out || total > capacity) return total;
    int32_t* at[13];
    for (int i = 0; i < 13; ++i) at[i] = out + offsets[i];
    struct Tile { int32_t seg, off; int64_t start; };
    std::vector<Tile> work;
    try {
        work.reserve((size_t)tiles);
    } catch (const std::exception&) {
        set_error("seq_step_fill: no memory for %lld query tiles", (long long)tiles);
        return SLLM_ENOMEM;
    }
    int32_t t = 0, first_tile = 0;
    for (int i = 0; i < nseg; ++i) {
        const int32_t slot = segments[4 * i], pos0 = segments[4 * i + 1], len = segments[4 * i + 2];
        at[3][i] = t; at[4][i] = len; at[5][i] = slot; at[6][i] = pos0; at[11][i] = first_tile;
        first_tile += (len + tile - 1) / tile;
        for (int32_t k = 0; k < len; ++k, ++t) {
            at[0][t] = tokens[t];
            at[1][t] = slot;
            at[2][t] = pos0 + k;
            at[12][t] = k ? tokens[t - 1] : segments[4 * i + 3];
        }
        for (int32_t off = 0; off < len; off += tile) work.push_back({i, off, (int64_t)pos0 + off});
    }
    // long tiles first: a tile's work grows with its last position; equal ones in the order of the batch
    std::sort(work.begin(), work.end(), [](const Tile& a, const Tile& b) {
        return a.start != b.start ? a.start > b.start : a.seg < b.seg;      // (two tiles of a segment never start at the same position)
    });
    for (int64_t i = 0; i < tiles; ++i) {
        at[7][i] = work[(size_t)i].seg;
        at[8][i] = work[(size_t)i].off;
    }
    at[9][0] = 0;
    std::copy(rows, rows + n_rows, at[9]);
    std::copy(kp->table.begin(), kp->table.end(), at[10]);
    return total;
}

}  // extern "C"
