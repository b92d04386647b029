// Decoded tokens' attention with a distance bias over whole pages (b200_decode_rows.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace b200 {

struct DecodeRows {      // arguments as in b200_biased_prompt_attn_ext
  void* out;
  const void* q; int64_t q_stride;
  const void* gate; int64_t gate_stride;
  const void* k_pool; const void* v_pool;
  const int32_t* block_tables; int table_stride;
  const int32_t* tiles;      // (first packed row, tokens, row of the block table) each
  const int32_t* tok_pos;
  const float* bias_lut; int lut_len;
  float scale, temp_coef; int temp_every;
  int H, G, block_size;
  float* ws;                 // (maximum, sum, output) per key range, tile, token and head; null: one CTA walks all keys
  int ws_tile, split_keys;   // tokens a tile has room for there, keys per range
};

// 0: launched.  1: not a shape of this kernel, nothing launched.
int decode_rows(const DecodeRows& A, int dk, int dv, int max_tile_tokens, int n_tiles, int n_splits, int dtype, cudaStream_t stream);

}  // namespace b200
