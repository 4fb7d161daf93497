// Attention over the paged cache for the rows of a prefill chunk.  Interface of attn_prefill.cu; see there for the design.
#pragma once
#include "common.cuh"
#include "token.cuh"

namespace ab {

// A run of consecutive positions of one sequence inside a chunk, at most one attention tile of them.
struct AttnTile { int32_t row, seq, pos, n_tok; };      // first chunk row, sequence, first position, positions

struct AttnPrefillArgs {
    float* qkv; uint32_t qkv_ld;                        // chunk rows: n_head query rows, n_kv key rows, n_kv value rows of head_dim each
    const float *q_norm, *k_norm; float eps;
    const float *cos_t, *sin_t; uint32_t n_pos;
    void* kv_pool; KvGeom geo; const int32_t* block_table;
    const int32_t *row_seq, *row_pos;                   // per chunk row
    const AttnTile* tiles; uint32_t n_tiles;            // cut for attn_prefill_tokens(...) positions each
    uint32_t n_rows, n_head, head_dim, layer, window;
    float scale, cap;
    float* out;                                         // [row][n_head * head_dim]
    uint32_t* err;
};

// Query rows per attention tile: the widest of 128 (head_dim <= 128: shared memory), 64 and 32 whose tiles still give every
// SM one.  A wide tile reads the cache less often; below one tile per SM the chunk's time is that of its longest tile, which
// a narrow tile, with more warps to each query row, gets through faster.  `positions`: rows of the chunk's sequences.
inline uint32_t attn_prefill_tokens(uint32_t group, uint32_t rows) { return rows / group; }     // positions per tile
inline uint32_t attn_prefill_rows(uint32_t positions, uint32_t group, uint32_t n_kv, uint32_t head_dim, uint32_t sms) {
    for (uint32_t rows = head_dim <= 128 ? 128 : 64; rows > 32; rows /= 2)
        if ((uint64_t)positions * group / rows * n_kv >= sms || rows / 2 < group) return rows;
    return 32;
}
// QK-norm + RoPE of the chunk's query rows (in place) and key rows, append of keys and values to the cache.
int launch_qkv_prep(const AttnPrefillArgs& a, bool kv_half, cudaStream_t stream, bool pdl);
// Causal (and windowed) soft-max attention of every chunk row over the cache, which already holds the chunk's rows.
int launch_attn_prefill(const AttnPrefillArgs& a, bool kv_half, uint32_t tile_rows, cudaStream_t stream, bool pdl);

}  // namespace ab
