// Launchers of b200_column_scan.cu, called by the C entry points of the recurrences; arguments as in b200_mixers.h, checked there.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace b200 {

struct ScanRows {   // where a step's inputs are; `stride` is theirs in elements
  const void* q;
  const void* k;    // gated: the forget gate's logits
  const void* v;
  int64_t stride;
};
struct ScanShape {
  int n_seqs, H, G, dk, dv;   // G: heads of q and k
};

int gated_column_scan(float* o, const ScanRows& in, const void* f_bias, const void* lower, float* state, const int32_t* seqs,
                      const ScanShape& n, int dtype, cudaStream_t stream);
int delta_column_scan(float* o, const ScanRows& in, const void* beta, int64_t beta_stride, const void* a, int64_t a_stride,
                      const void* dt_bias, const void* a_log, bool per_channel, float* state, const int32_t* seqs,
                      const ScanShape& n, float unit_eps, float q_scale, int dtype, cudaStream_t stream);
int retention_column_scan(float* o, const ScanRows& in, const float* decay, float k_scale, float* state, const int32_t* seqs,
                          const ScanShape& n, int dtype, cudaStream_t stream);

}  // namespace b200
