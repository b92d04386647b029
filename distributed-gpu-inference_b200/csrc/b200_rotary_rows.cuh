// Launchers of b200_rotary_rows.cu: false where the rows cannot be moved in 16-byte pieces (nothing launched).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace b200 {

struct QkRows {     // arguments as in b200_qknorm_rotary_append_ext2
  void* q; int64_t q_stride;
  const void* k; int64_t k_stride;
  const void* v; int64_t v_stride;
  const void* qw; const void* kw;
  int unit_norm; float eps;
  const double* freqs; int rot_dims, interleaved;
  void* k_pool; void* v_pool;
  const int64_t* slot_mapping; const int32_t* tok_pos;
  int n_tok, H, G, Gv, dk, dv, block_size;
};
struct LatentRows {     // as in b200_latent_rotary_append_ext
  const void* q; int64_t q_tok_stride, q_head_stride;
  void* q_out; int64_t qo_tok_stride, qo_head_stride;
  const void* dkv; int64_t dkv_stride;
  const void* w_c; float eps;
  const double* freqs; float gain; int rot_dims, interleaved;
  void* pool;
  const int64_t* slot_mapping; const int32_t* tok_pos;
  int n_tok, H, dr, rank;
};

bool qk_rows(const QkRows& A, int dtype, cudaStream_t stream);
bool latent_rows(const LatentRows& A, int dtype, cudaStream_t stream);

}  // namespace b200
