// Launchers of b200_tile_attn.cu (the C entry point b200_tile_attn checks the arguments and runs the merge of key splits).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace b200 {

constexpr int kTileRows = 128;   // rows of a product; a tile has one or two times as many (tile_attn_rows)

struct TileAttn {
  void* out; int64_t out_tok_stride, out_head_stride;
  const void* q; int64_t q_tok_stride, q_head_stride;
  const void* gate; int64_t gate_stride;
  const void* k_pool; const void* v_pool;
  const int32_t* block_tables; int table_stride;
  const int32_t* tiles; const int32_t* tok_pos;
  const float* sink;
  const float* bias_lut; int lut_len;        // distance biases [H][lut_len], or null
  float* ws;                                 // key splits: [split][tile][token of the tile][H][dv + 2]
  int H, G, block_size, v_row, v_div;
  int window, keep_first, chunk;
  int gate_dim, out_f32, out_vec;            // gates per channel: the value size; 16-byte stores possible
  float scale, softcap, temp_coef;
  int temp_every;
  int boxes, q_boxes;                        // set by the launcher: pages, and the queries of full tiles, come by the copy engine
  int tile0, n_tiles;                        // and the first tile of a launch, and how many the call has
};

bool tile_attn_supported(int H, int G, int dk, int dv, bool alias, bool bias, int dtype);
int tile_attn_rows(int rep, int G, int dk, int n_tokens, bool heavy, bool boxes);   // heavy: distance biases or a soft cap
int tile_attn_splits(int n_tiles, int key_tiles, int G, int dk, int rows, int64_t live_rows);   // live: tokens x heads of all tiles
int tile_attn_launch(const TileAttn& A, int dk, int dv, bool alias, int rows, int n_tiles, int n_splits, int dtype, cudaStream_t stream);

}  // namespace b200
