// One Llama decoder layer of a decode step (one new token per sequence) in five launches from one call, for up to 32 sequences:
//
//   norm + q | k | v      y = T(w T(x rsqrt(mean x^2 + eps))) in registers, the three projections side by side; one more CTA makes the
//                         RoPE tables when the caller has none
//   attention             b200_rope_append_decode_attn: RoPE, append and paged attention
//   output + residual     h = T(x + T(Wo a))
//   norm + gate, up       T(T(silu(T(Wg y))) T(Wu y))
//   down + residual       T(h + T(Wd act))
//
// Every result is rounded to the storage type where the separate launches round it.
//
// The projections (skinny_kernel): a CTA has 16 output rows (two times 16 for gate and up), its eight warps every eighth block of 32
// inputs.  Weights are the A operand of m16n8k16, the sequences' rows B; a lane reads 16 consecutive bytes of a weight row and of an input
// row, and since any order of the contraction will do as long as both sides have the same, these are its fragments of two products as
// they come.  Weights are asked for before the launch in front has finished (they do not depend on it), inputs after.
//
// What bounds it: at the widths of small models (512: 6 MB of weights per layer) the launches and their latencies, not the bytes.  B200,
// bf16, width 512, batch 4: 13 launches a layer from Python took 250 us of host time, this call with the checks before it 58 us.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "b200_attn.cuh"
#include "b200_common.cuh"
#include "b200_tma_common.cuh"

namespace b200 {
namespace {

constexpr int kWarps = 8;
constexpr int kMaxBatch = 32;

struct Skinny {
  void* out; int64_t out_stride;
  const void* x; int64_t x_stride;
  const void* w[3];         // [rows[i], K], contiguous
  int rows[3];
  const void* norm; float eps;
  const void* resid; int64_t resid_stride;
  int B, K;
  // RoPE tables, by the last CTA
  void* cos; void* sin;
  const int64_t* pos; const float* inv_freq;
  int half; float scaling;
};

template <typename T>
union Piece {
  uint4 raw;
  uint32_t u[4];
  T e[8];
};
template <typename T>
__device__ __forceinline__ Piece<T> piece(const T* p) {
  Piece<T> r;
  r.raw = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <typename T>
__device__ __forceinline__ Piece<T> weight_piece(const T* p) {     // read once: not into L1
  Piece<T> r;
  const int4 v = ld_stream16(p);
  r.raw = make_uint4(v.x, v.y, v.z, v.w);
  return r;
}

// NB: tiles of eight sequences.  DEP: launched as a programmatic dependent of the launch in front.
template <typename T, int NB, bool NORM, bool GATED, bool DEP>
__global__ void __launch_bounds__(32 * kWarps)
skinny_kernel(const Skinny A) {
  constexpr int NM = GATED ? 2 : 1, kLd = 8 * NB + 1, kAhead = 2;
  __shared__ float red[kWarps][NM][16][kLd];
  __shared__ float squares[kWarps][8 * NB];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  if (NORM && A.cos && blockIdx.x == gridDim.x - 1) {
    for (int i = threadIdx.x; i < A.B * A.half; i += 32 * kWarps) {
      const int n = i / A.half, j = i - n * A.half;
      const float angle = __fmul_rn(static_cast<float>(A.pos[n]), A.inv_freq[j]);
      T* cs = static_cast<T*>(A.cos) + n * 2 * A.half + j;
      T* sn = static_cast<T*>(A.sin) + n * 2 * A.half + j;
      cs[0] = cs[A.half] = Cvt<T>::from_f32(__fmul_rn(cosf(angle), A.scaling));
      sn[0] = sn[A.half] = Cvt<T>::from_f32(__fmul_rn(sinf(angle), A.scaling));
    }
    return;
  }
  const int col0 = 16 * blockIdx.x, K = A.K, blocks = K / 32;
  const T* wp[NM];
  if constexpr (GATED) {
    wp[0] = static_cast<const T*>(A.w[0]) + static_cast<int64_t>(col0 + r) * K + 8 * c;
    wp[NM - 1] = static_cast<const T*>(A.w[1]) + static_cast<int64_t>(col0 + r) * K + 8 * c;
  } else {
    int row0 = col0, which = 0;
    if (row0 >= A.rows[0]) row0 -= A.rows[0], which = 1;
    if (which == 1 && row0 >= A.rows[1]) row0 -= A.rows[1], which = 2;
    wp[0] = static_cast<const T*>(A.w[which]) + static_cast<int64_t>(row0 + r) * K + 8 * c;
  }
  auto weights = [&](Piece<T> (&w)[NM][2], int b) {
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      w[m][0] = weight_piece(wp[m] + 32 * b);
      w[m][1] = weight_piece(wp[m] + 32 * b + 8 * static_cast<int64_t>(K));
    }
  };
  Piece<T> w[kAhead][NM][2];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) {
    if (warp + kWarps * i < blocks) weights(w[i], warp + kWarps * i);
  }
  if constexpr (DEP) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
  }
  const T* xp[NB];
#pragma unroll
  for (int t = 0; t < NB; ++t) xp[t] = static_cast<const T*>(A.x) + min(8 * t + r, A.B - 1) * A.x_stride + 8 * c;
  float inv[NB];
  if constexpr (NORM) {
    float ss[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) ss[t] = 0.f;
    for (int b = warp; b < blocks; b += kWarps) {
#pragma unroll
      for (int t = 0; t < NB; ++t) {
        const Piece<T> x = piece(xp[t] + 32 * b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float f = Cvt<T>::to_f32(x.e[i]);
          ss[t] = fmaf(f, f, ss[t]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      ss[t] += __shfl_xor_sync(0xffffffffu, ss[t], 1);
      ss[t] += __shfl_xor_sync(0xffffffffu, ss[t], 2);
      if (c == 0) squares[warp][8 * t + r] = ss[t];
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < kWarps; ++i) sum += squares[i][8 * t + r];
      inv[t] = rsqrtf(sum * (1.0f / static_cast<float>(K)) + A.eps);
    }
  }
  float acc[NM][NB][4];
#pragma unroll
  for (int m = 0; m < NM; ++m) {
#pragma unroll
    for (int t = 0; t < NB; ++t) {
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][t][i] = 0.f;
    }
  }
  auto products = [&](const Piece<T> (&w)[NM][2], int b) {
    Piece<T> g;
    if constexpr (NORM) g = piece(static_cast<const T*>(A.norm) + 32 * b + 8 * c);
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      Piece<T> x = piece(xp[t] + 32 * b);
      if constexpr (NORM) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const T n = Cvt<T>::from_f32(__fmul_rn(Cvt<T>::to_f32(x.e[i]), inv[t]));
          x.e[i] = Cvt<T>::from_f32(__fmul_rn(Cvt<T>::to_f32(g.e[i]), Cvt<T>::to_f32(n)));
        }
      }
#pragma unroll
      for (int m = 0; m < NM; ++m) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const uint32_t a[4] = {w[m][0].u[2 * s], w[m][1].u[2 * s], w[m][0].u[2 * s + 1], w[m][1].u[2 * s + 1]};
          tma::Mma<T>::run(acc[m][t], a, x.u[2 * s], x.u[2 * s + 1]);
        }
      }
    }
  };
  for (int b = warp; b < blocks; b += kAhead * kWarps) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int now = b + kWarps * i, next = now + kAhead * kWarps;
      if (now < blocks) {
        products(w[i], now);
        if (next < blocks) weights(w[i], next);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < NM; ++m) {
#pragma unroll
    for (int t = 0; t < NB; ++t) {
#pragma unroll
      for (int i = 0; i < 4; ++i) red[warp][m][r + 8 * (i >> 1)][8 * t + 2 * c + (i & 1)] = acc[m][t][i];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * A.B; i += 32 * kWarps) {
    const int row = i & 15, b = i >> 4;
    float sum[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      sum[m] = 0.f;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) sum[m] += red[k][m][row][b];
    }
    T y = Cvt<T>::from_f32(sum[0]);
    if constexpr (GATED) {
      const float g = Cvt<T>::to_f32(y);
      const T s = Cvt<T>::from_f32(g / (1.0f + expf(-g)));
      y = Cvt<T>::from_f32(__fmul_rn(Cvt<T>::to_f32(s), Cvt<T>::to_f32(Cvt<T>::from_f32(sum[NM - 1]))));
    } else if constexpr (!NORM) {
      y = Cvt<T>::from_f32(__fadd_rn(Cvt<T>::to_f32(static_cast<const T*>(A.resid)[b * A.resid_stride + col0 + row]), Cvt<T>::to_f32(y)));
    }
    static_cast<T*>(A.out)[b * A.out_stride + col0 + row] = y;
  }
}

template <typename T, bool NORM, bool GATED, bool DEP>
int launch_skinny(const Skinny& A, cudaStream_t stream) {
  const int rows = GATED ? A.rows[0] : A.rows[0] + A.rows[1] + A.rows[2];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows / 16 + (NORM && A.cos ? 1 : 0));
  cfg.blockDim = dim3(32 * kWarps);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = DEP ? 1 : 0;
  auto go = [&](auto kern) {
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, A);
    return e == cudaSuccess ? 0 : fail(static_cast<int>(e), "b200_llama_decode_layer: %s", cudaGetErrorString(e));
  };
  if (A.B <= 8) return go(skinny_kernel<T, 1, NORM, GATED, DEP>);
  if (A.B <= 16) return go(skinny_kernel<T, 2, NORM, GATED, DEP>);
  return go(skinny_kernel<T, 4, NORM, GATED, DEP>);
}

int64_t up16(int64_t n) { return (n + 15) / 16 * 16; }
struct Scratch {
  int64_t qkv, attn, h, act, cos, sin, split, total;      // bytes from the start
};
Scratch scratch_of(int B, int W, int ff, int Hq, int Hkv, int D, size_t split_bytes) {
  Scratch s;
  int64_t at = 0;
  auto take = [&](int64_t bytes) {
    const int64_t here = at;
    at += up16(bytes);
    return here;
  };
  s.qkv = take(2ll * B * (Hq + 2 * Hkv) * D);
  s.attn = take(2ll * B * Hq * D);
  s.h = take(2ll * B * W);
  s.act = take(2ll * B * ff);
  s.cos = take(2ll * B * D);
  s.sin = take(2ll * B * D);
  s.split = take(static_cast<int64_t>(split_bytes));
  s.total = at;
  return s;
}
int splits_of(int B, int Hq, int Hkv, int D, int block_size, int max_context_len, int num_splits, int dtype) {
  return num_splits > 0 ? num_splits : std::max(1, b200_paged_decode_attn_plan(B, Hq, Hkv, D, block_size, max_context_len, dtype));
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int b200_llama_decode_layer_supported(int B, int W, int ff, int Hq, int Hkv, int D, int block_size, int dtype) {
  return (dtype == B200_DTYPE_F16 || dtype == B200_DTYPE_BF16) && B >= 1 && B <= kMaxBatch && W > 0 && W % 32 == 0 && ff > 0 && ff % 32 == 0 &&
         Hkv > 0 && Hq > 0 && Hq % Hkv == 0 && Hq / Hkv <= 8 && (D == 64 || D == 128) && block_size == 16;
}

size_t b200_llama_decode_layer_workspace(int B, int W, int ff, int Hq, int Hkv, int D, int block_size, int max_context_len, int num_splits,
                                         int dtype) {
  if (!b200_llama_decode_layer_supported(B, W, ff, Hq, Hkv, D, block_size, dtype)) return 0;
  const int splits = splits_of(B, Hq, Hkv, D, block_size, max_context_len, num_splits, dtype);
  return static_cast<size_t>(scratch_of(B, W, ff, Hq, Hkv, D, splits > 1 ? b200_paged_decode_attn_workspace(B, Hq, D, splits) : 0).total);
}

int b200_llama_decode_layer(void* h_out, const void* x, int64_t x_stride, const void* norm1, float eps1, const void* wq, const void* wk,
                            const void* wv, const void* wo, const void* norm2, float eps2, const void* wg, const void* wu, const void* wd,
                            const int64_t* pos, const float* inv_freq, float rope_scaling, const void* cos_table, const void* sin_table,
                            void* k_pool, void* v_pool, const int32_t* block_tables, int table_stride, const int32_t* context_lens, int B,
                            int W, int ff, int Hq, int Hkv, int D, int block_size, int64_t max_blocks, int max_context_len, int num_splits,
                            void* workspace, size_t workspace_bytes, int dtype, unsigned attn_flags, void* stream) {
  const char* name = "b200_llama_decode_layer";
  if (!b200_llama_decode_layer_supported(B, W, ff, Hq, Hkv, D, block_size, dtype)) return fail(B200_ESHAPE, "%s: sizes or dtype not served", name);
  const bool tables = cos_table && sin_table;
  if (!h_out || !x || !norm1 || !wq || !wk || !wv || !wo || !norm2 || !wg || !wu || !wd || !workspace || (!tables && (!pos || !inv_freq)))
    return fail(B200_EINVAL, "%s: null pointer", name);
  for (const void* p : {x, norm1, wq, wk, wv, wo, norm2, wg, wu, wd, static_cast<const void*>(workspace)}) {
    if (!aligned16(p)) return fail(B200_EINVAL, "%s: operands must be 16-byte aligned", name);
  }
  if (x_stride % 8 || x_stride < W) return fail(B200_EINVAL, "%s: row stride %lld", name, static_cast<long long>(x_stride));
  const int splits = splits_of(B, Hq, Hkv, D, block_size, max_context_len, num_splits, dtype);
  const size_t split_bytes = splits > 1 ? b200_paged_decode_attn_workspace(B, Hq, D, splits) : 0;
  const Scratch at = scratch_of(B, W, ff, Hq, Hkv, D, split_bytes);
  if (workspace_bytes < static_cast<size_t>(at.total)) return fail(B200_ENOSPC, "%s: workspace of %zu bytes, %lld needed", name, workspace_bytes, static_cast<long long>(at.total));
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  const int nq = Hq * D, nk = Hkv * D, nqkv = nq + 2 * nk;
  auto st = static_cast<cudaStream_t>(stream);
  auto run = [&](auto* tag) -> int {
    using T = std::remove_pointer_t<decltype(tag)>;
    Skinny a{};
    a.out = ws + at.qkv, a.out_stride = nqkv, a.x = x, a.x_stride = x_stride;
    a.w[0] = wq, a.w[1] = wk, a.w[2] = wv, a.rows[0] = nq, a.rows[1] = a.rows[2] = nk;
    a.norm = norm1, a.eps = eps1, a.B = B, a.K = W;
    if (!tables) {
      a.cos = ws + at.cos, a.sin = ws + at.sin, a.pos = pos, a.inv_freq = inv_freq, a.half = D / 2, a.scaling = rope_scaling;
    }
    if (int rc = launch_skinny<T, true, false, false>(a, st)) return rc;
    const T* qkv = reinterpret_cast<const T*>(ws + at.qkv);
    if (int rc = b200_rope_append_decode_attn(ws + at.attn, qkv, nqkv, qkv + nq, nqkv, qkv + nq + nk, nqkv, tables ? cos_table : ws + at.cos,
                                              tables ? sin_table : ws + at.sin, k_pool, v_pool, block_tables, table_stride, context_lens, B, Hq,
                                              Hkv, D, block_size, max_blocks, static_cast<float>(1.0 / std::sqrt(static_cast<double>(D))), max_context_len, splits,
                                              split_bytes ? ws + at.split : nullptr, split_bytes, dtype, attn_flags, stream))
      return rc;
    Skinny o{};
    o.out = ws + at.h, o.out_stride = W, o.x = ws + at.attn, o.x_stride = nq, o.w[0] = wo, o.rows[0] = W;
    o.resid = x, o.resid_stride = x_stride, o.B = B, o.K = nq;
    if (int rc = launch_skinny<T, false, false, true>(o, st)) return rc;
    Skinny g{};
    g.out = ws + at.act, g.out_stride = ff, g.x = ws + at.h, g.x_stride = W, g.w[0] = wg, g.w[1] = wu, g.rows[0] = ff;
    g.norm = norm2, g.eps = eps2, g.B = B, g.K = W;
    if (int rc = launch_skinny<T, true, true, true>(g, st)) return rc;
    Skinny d{};
    d.out = h_out, d.out_stride = W, d.x = ws + at.act, d.x_stride = ff, d.w[0] = wd, d.rows[0] = W;
    d.resid = ws + at.h, d.resid_stride = W, d.B = B, d.K = ff;
    return launch_skinny<T, false, false, true>(d, st);
  };
  return dtype == B200_DTYPE_F16 ? run(static_cast<__half*>(nullptr)) : run(static_cast<__nv_bfloat16*>(nullptr));
}

}  // extern "C"
