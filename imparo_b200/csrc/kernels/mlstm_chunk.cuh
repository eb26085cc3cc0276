// What mlstm.cu calls of mlstm_chunk.cu.
#pragma once
#include "common.cuh"

namespace imparo {

struct MlstmProducts {
    const float* proj;      // float32 rows of `stride` floats
    size_t stride;
    int q_off, k_off, v_off, i_off, f_off;
    const float* i_bias;    // [heads]
    const float* f_bias;    // [heads]
    float cap, q_scale;
    const int* item_row_start; const int* item_slot;
    int n_items, n_slots, heads, dim, vdim, vblocks;
    float* chunk_S;         // [chunks, heads, dim, vdim]
    float* chunk_n;         // [chunks, heads, vblocks, dim]
    float* chunk_mb;        // [chunks, heads, vblocks, 3]: the chunk's own maximum, its total b, the maximum it starts from
    float* state_m;         // [slots, heads, vblocks]
    float* out;             // [tokens, heads * vdim]
};

constexpr int MLSTM_PRODUCTS_CHUNK = 64;
// sizes and alignments the products take
bool mlstm_products_take(const MlstmProducts& p);
// every chunk's own state and maximum; the outputs of every chunk from the state the scan left for it
int mlstm_products_local(const MlstmProducts& p, int max_chunks, cudaStream_t stream);
int mlstm_products_out(const MlstmProducts& p, int max_chunks, cudaStream_t stream);

}  // namespace imparo
