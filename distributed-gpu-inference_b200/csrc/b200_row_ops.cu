// Row-wise pieces of the ragged-batch mixers: norms, residual updates, value preparation, activations, and what moves rows to experts
// and back.  All are bound by the bytes of their rows, so a row is read once, in 16-byte pieces, and stays in registers between the
// passes over it; rows that cannot be read that way (sizes or addresses off the 16-byte grid) take the element-wise form.
//
//   offset RMS norm            y = x * rsqrt(mean(x^2) + eps) * (1 + w)            fp32 in, storage dtype out
//   post-norm residual update  x += m * norm(y; w_post), optionally followed by the next sublayer's input norm
//   value prep + paged append  per-head unit-RMS values, optional mix with an earlier layer's values, K/V scatter
//   per-head RMS norm          of a recurrence's fp32 read-outs, with a weight, a sigmoid or SiLU gate and a factor
//   PolyNorm activation        a N(z) + b N(z^2) + c N(z^3) + e over a token's feed-forward row
//   expert order               a stable sort of (token, choice) pairs by expert in one CTA, with the experts' row offsets
//   input-scaled expert rows, clamped GLU, combine
//
// Measured on B200 (bf16), element-wise -> this: post-norm residual with the next norm, 2600 rows of 1024: 15.1 -> 7.7 us; PolyNorm, 2600 x
// 4096: 26.4 -> 11.5; value prep, 16384 tokens of 4 heads of 128 + 128: 52 -> 34; clamped GLU, 8198 x 1024: 28.5 -> 12.6; expert rows in
// 14.5 -> 6.6, out 12.1 -> 7.2; expert order of 8198 pairs: 12.6 (sort, count and inverse by library calls: 75 and a wait on the host).
#include <algorithm>
#include <type_traits>

#include "../../include/b200_mixers.h"
#include "b200_common.cuh"

namespace b200 {
namespace {

template <typename F>
int rows_by_dtype(int dtype, const char* name, F&& f) {
  switch (dtype) {
    case B200_DTYPE_F16:
      return f(static_cast<__half*>(nullptr));
    case B200_DTYPE_BF16:
      return f(static_cast<__nv_bfloat16*>(nullptr));
    case B200_DTYPE_F32:
      return f(static_cast<float*>(nullptr));
    default:
      return fail(B200_EINVAL, "%s: unsupported dtype %d", name, dtype);
  }
}

// N consecutive elements as fp32 (N * sizeof(T) a multiple of 8: 8- or 16-byte accesses)
template <int N, typename T>
__device__ __forceinline__ void get(float (&d)[N], const T* p) {
  if constexpr (N * sizeof(T) == 8) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < N; ++i) d[i] = Cvt<T>::to_f32(e[i]);
  } else {
    constexpr int E = 16 / sizeof(T);
#pragma unroll
    for (int j = 0; j < N / E; ++j) {
      const uint4 raw = *reinterpret_cast<const uint4*>(p + j * E);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < E; ++i) d[j * E + i] = Cvt<T>::to_f32(e[i]);
    }
  }
}
template <int N, typename T>
__device__ __forceinline__ void put(T* p, const float (&d)[N]) {
  if constexpr (N * sizeof(T) == 8) {
    uint2 raw;
    T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = Cvt<T>::from_f32(d[i]);
    *reinterpret_cast<uint2*>(p) = raw;
  } else {
    constexpr int E = 16 / sizeof(T);
#pragma unroll
    for (int j = 0; j < N / E; ++j) {
      uint4 raw;
      T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
      for (int i = 0; i < E; ++i) e[i] = Cvt<T>::from_f32(d[j * E + i]);
      *reinterpret_cast<uint4*>(p + j * E) = raw;
    }
  }
}

// Sum over the WPR warps that share a row (one row per warp, or one per CTA); `red` holds WPR floats per call.
template <int WPR>
__device__ __forceinline__ float row_sum(float v, float* red) {
  v = warp_sum(v);
  if constexpr (WPR == 1) return v;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < WPR; ++w) t += red[w];
  return t;
}

// squares of a piece, added pairwise (three roundings deep instead of eight)
__device__ __forceinline__ float squares(const float (&d)[8]) {
  const float a = fmaf(d[0], d[0], d[1] * d[1]), b = fmaf(d[2], d[2], d[3] * d[3]);
  const float c = fmaf(d[4], d[4], d[5] * d[5]), e = fmaf(d[6], d[6], d[7] * d[7]);
  return (a + b) + (c + e);
}

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.f);
}

// A row over WPR warps, NCH pieces of eight elements per lane: by its width alone, so that a row's sums do not depend on the step.
// Rows of up to 1024 elements go to one warp each (no barrier).
template <typename F>
bool by_row_shape(int width, F&& f) {
  auto go = [&](auto wpr, auto nch) { f(wpr, nch); };
  using std::integral_constant;
  if (width <= 512) go(integral_constant<int, 1>{}, integral_constant<int, 2>{});
  else if (width <= 1024) go(integral_constant<int, 1>{}, integral_constant<int, 4>{});
  else if (width <= 2048) go(integral_constant<int, 4>{}, integral_constant<int, 2>{});
  else if (width <= 4096) go(integral_constant<int, 4>{}, integral_constant<int, 4>{});
  else if (width <= 8192) go(integral_constant<int, 8>{}, integral_constant<int, 4>{});
  else if (width <= 16384) go(integral_constant<int, 8>{}, integral_constant<int, 8>{});
  else return false;
  return true;
}
template <int WPR>
struct RowCta {
  static constexpr int kWarps = WPR == 1 ? 4 : WPR;      // per CTA
  static constexpr int kNT = 32 * kWarps;
  static unsigned grid(int64_t rows) { return static_cast<unsigned>(WPR == 1 ? (rows + 3) / 4 : rows); }
};
template <int WPR>
__device__ __forceinline__ int64_t my_row() {
  return WPR == 1 ? static_cast<int64_t>(blockIdx.x) * 4 + (threadIdx.x >> 5) : blockIdx.x;
}
template <int WPR>
__device__ __forceinline__ int my_piece(int c) {       // first element of the lane's piece c
  return ((WPR == 1 ? threadIdx.x & 31 : threadIdx.x) + c * 32 * WPR) * 8;
}

// ---- offset RMS norm ------------------------------------------------------------------------------------------
template <typename T, int WPR, int NCH>
__global__ void __launch_bounds__(RowCta<WPR>::kNT)
offset_rmsnorm_rows(T* __restrict__ out, const float* __restrict__ x, const T* __restrict__ w, float eps, int64_t rows, int width) {
  __shared__ float red[8];
  const int64_t row = my_row<WPR>();
  if (row >= rows) return;
  float v[NCH][8], ss = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < width) {
      get(v[c], x + row * width + i);
      ss += squares(v[c]);
    }
  }
  const float inv = rsqrtf(row_sum<WPR>(ss, red) / static_cast<float>(width) + eps);
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < width) {
      float g[8];
      get(g, w + i);
#pragma unroll
      for (int u = 0; u < 8; ++u) v[c][u] = v[c][u] * inv * (1.0f + g[u]);
      put(out + row * width + i, v[c]);
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(256)
offset_rmsnorm_kernel(T* __restrict__ out, const float* __restrict__ x, const T* __restrict__ w, float eps, int width) {
  __shared__ float red[32];
  const float* xr = x + static_cast<int64_t>(blockIdx.x) * width;
  float ss = 0.f;
  for (int i = threadIdx.x; i < width; i += blockDim.x) ss = fmaf(xr[i], xr[i], ss);
  const float inv = rsqrtf(block_sum(ss, red) / static_cast<float>(width) + eps);
  T* orow = out + static_cast<int64_t>(blockIdx.x) * width;
  for (int i = threadIdx.x; i < width; i += blockDim.x)
    orow[i] = Cvt<T>::from_f32(xr[i] * inv * (1.0f + Cvt<T>::to_f32(w[i])));
}

// ---- x += mult * norm(y; w_post); optionally out_next = norm(x; w_next) ------------------------------------------
template <typename T, typename Y, int WPR, int NCH>
__global__ void __launch_bounds__(RowCta<WPR>::kNT)
postnorm_residual_rows(float* __restrict__ x, const Y* __restrict__ y, int64_t y_stride, const T* __restrict__ w_post, float mult,
                       const T* __restrict__ w_next, T* __restrict__ out_next, float eps, int64_t rows, int width) {
  __shared__ float red[16];
  const int64_t row = my_row<WPR>();
  if (row >= rows) return;
  float v[NCH][8], r[NCH][8], ss = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < width) {
      get(v[c], y + row * y_stride + i);
      get(r[c], x + row * width + i);
      ss += squares(v[c]);
    }
  }
  const float inv = rsqrtf(row_sum<WPR>(ss, red) / static_cast<float>(width) + eps);
  float sx = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < width) {
      float g[8];
      get(g, w_post + i);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float n = v[c][u] * inv * (1.0f + g[u]);
        r[c][u] += mult * n;
      }
      sx += squares(r[c]);
      put(x + row * width + i, r[c]);
    }
  }
  if (w_next == nullptr) return;
  const float inv2 = rsqrtf(row_sum<WPR>(sx, red + 8) / static_cast<float>(width) + eps);
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < width) {
      float g[8];
      get(g, w_next + i);
#pragma unroll
      for (int u = 0; u < 8; ++u) r[c][u] = r[c][u] * inv2 * (1.0f + g[u]);
      put(out_next + row * width + i, r[c]);
    }
  }
}
// element-wise form: the updated row is kept in shared memory between the update and the second norm
template <typename T, typename Y>
__global__ void __launch_bounds__(256)
postnorm_residual_kernel(float* __restrict__ x, const Y* __restrict__ y, int64_t y_stride, const T* __restrict__ w_post,
                         float mult, const T* __restrict__ w_next, T* __restrict__ out_next, float eps, int width) {
  extern __shared__ float row_s[];
  __shared__ float red[32];
  const Y* yr = y + static_cast<int64_t>(blockIdx.x) * y_stride;
  float* xr = x + static_cast<int64_t>(blockIdx.x) * width;
  float ss = 0.f;
  for (int i = threadIdx.x; i < width; i += blockDim.x) {
    const float v = Cvt<Y>::to_f32(yr[i]);
    ss = fmaf(v, v, ss);
  }
  const float inv = rsqrtf(block_sum(ss, red) / static_cast<float>(width) + eps);
  float sx = 0.f;
  for (int i = threadIdx.x; i < width; i += blockDim.x) {
    const float n = Cvt<Y>::to_f32(yr[i]) * inv * (1.0f + Cvt<T>::to_f32(w_post[i]));
    const float v = xr[i] + mult * n;
    xr[i] = v;
    row_s[i] = v;
    sx = fmaf(v, v, sx);
  }
  if (w_next == nullptr) return;
  const float inv2 = rsqrtf(block_sum(sx, red) / static_cast<float>(width) + eps);
  T* orow = out_next + static_cast<int64_t>(blockIdx.x) * width;
  for (int i = threadIdx.x; i < width; i += blockDim.x)
    orow[i] = Cvt<T>::from_f32(row_s[i] * inv2 * (1.0f + Cvt<T>::to_f32(w_next[i])));
}

// ---- value prep + K/V append ------------------------------------------------------------------------------------
// One warp per (token, kv head).  v <- v / rms(v); with `v_prev` the stored value is (1 - lam) v + lam v_prev.  The stored value also
// goes to `v_keep` (for later layers of the same step) when given.  N elements per access (four, or one where rows are not aligned).
template <typename T, int N>
__global__ void __launch_bounds__(256)
value_prep_append_kernel(const T* __restrict__ k, int64_t k_stride, const T* __restrict__ v, int64_t v_stride,
                         const T* __restrict__ v_prev, T* __restrict__ v_keep, float lam, float eps,
                         T* __restrict__ k_pool, T* __restrict__ v_pool, const int64_t* __restrict__ slot_mapping,
                         int64_t n_tok, int G, int dk, int dv, int block_size, int64_t max_blocks) {
  const int64_t pair = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int64_t tok = pair / G;
  const int g = static_cast<int>(pair - tok * G), lane = threadIdx.x & 31;
  if (tok >= n_tok) return;
  const int64_t slot = slot_mapping[tok];
  const int64_t blk = slot >= 0 ? slot / block_size : -1;
  const bool store = blk >= 0 && blk < max_blocks;
  const int64_t at = store ? (blk * G + g) * block_size + (slot - blk * block_size) : 0;
  auto load = [](float (&d)[N], const T* p) {
    if constexpr (N == 1) d[0] = Cvt<T>::to_f32(p[0]);
    else get(d, p);
  };
  auto save = [](T* p, const float (&d)[N]) {
    if constexpr (N == 1) p[0] = Cvt<T>::from_f32(d[0]);
    else put(p, d);
  };
  const T* vr = v + tok * v_stride + g * dv;
  float ss = 0.f;
  for (int c = lane * N; c < dv; c += 32 * N) {
    float f[N];
    load(f, vr + c);
#pragma unroll
    for (int u = 0; u < N; ++u) ss = fmaf(f[u], f[u], ss);
  }
  const float inv = rsqrtf(warp_sum(ss) / static_cast<float>(dv) + eps);
  for (int c = lane * N; c < dv; c += 32 * N) {
    float f[N];
    load(f, vr + c);
#pragma unroll
    for (int u = 0; u < N; ++u) f[u] *= inv;
    if (v_prev) {
      float o[N];
      load(o, v_prev + (tok * G + g) * dv + c);
#pragma unroll
      for (int u = 0; u < N; ++u) f[u] = (1.0f - lam) * f[u] + lam * o[u];
    }
    if (store) save(v_pool + at * dv + c, f);
    if (v_keep) save(v_keep + (tok * G + g) * dv + c, f);
  }
  if (store) {
    for (int c = lane * N; c < dk; c += 32 * N) {
      const T* src = k + tok * k_stride + g * dk + c;
      T* dst = k_pool + at * dk + c;
      if constexpr (N == 1) {
        dst[0] = src[0];
      } else if constexpr (N * sizeof(T) == 8) {
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(src);
      } else {
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
      }
    }
  }
}

// The same in 16-byte pieces, LPR lanes per row of 8 LPR values and kPrepRows rows per lane under way at once: a warp per row with 8-byte
// accesses, values read twice, took
// 24.5 us for 16384 x 4 rows of 128 + 128 (67 MB), this 10.3; 592 x 4 rows 2.75 -> 2.5.
constexpr int kPrepRows = 2;
template <typename T, int LPR>
__global__ void __launch_bounds__(256)
value_prep_rows(const T* __restrict__ k, int64_t k_stride, const T* __restrict__ v, int64_t v_stride, const T* __restrict__ v_prev,
                T* __restrict__ v_keep, float lam, float eps, T* __restrict__ k_pool, T* __restrict__ v_pool,
                const int64_t* __restrict__ slot_mapping, int64_t rows, int G, int dk, int block_size, int64_t max_blocks) {
  constexpr int kPass = 32 / LPR, DV = 8 * LPR;
  const int lane = threadIdx.x & 31, c = 8 * (lane % LPR);
  const int64_t row0 = (static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5)) * (kPrepRows * kPass) + lane / LPR;
  float f[kPrepRows][8];
  uint4 key[kPrepRows], old[kPrepRows];
  int64_t tok[kPrepRows], at[kPrepRows];
  int g[kPrepRows];
#pragma unroll
  for (int r = 0; r < kPrepRows; ++r) {
    const int64_t row = min(row0 + r * kPass, rows - 1);
    tok[r] = static_cast<uint32_t>(row) / static_cast<uint32_t>(G);
    g[r] = static_cast<int>(row - tok[r] * G);
    get(f[r], v + tok[r] * v_stride + g[r] * DV + c);
    if (c < dk) key[r] = *reinterpret_cast<const uint4*>(k + tok[r] * k_stride + g[r] * dk + c);
    if (v_prev) old[r] = *reinterpret_cast<const uint4*>(v_prev + row * DV + c);
    const int64_t slot = slot_mapping[tok[r]], blk = slot >= 0 ? slot / block_size : -1;
    at[r] = blk >= 0 && blk < max_blocks ? (blk * G + g[r]) * block_size + (slot - blk * block_size) : -1;
  }
#pragma unroll
  for (int r = 0; r < kPrepRows; ++r) {
    float ss = squares(f[r]);
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const int64_t row = row0 + r * kPass;
    if (row >= rows) continue;
    const float inv = rsqrtf(ss / static_cast<float>(DV) + eps);
#pragma unroll
    for (int u = 0; u < 8; ++u) f[r][u] *= inv;
    if (v_prev) {
      const T* e = reinterpret_cast<const T*>(&old[r]);
#pragma unroll
      for (int u = 0; u < 8; ++u) f[r][u] = (1.0f - lam) * f[r][u] + lam * Cvt<T>::to_f32(e[u]);
    }
    if (v_keep) put(v_keep + row * DV + c, f[r]);
    if (at[r] < 0) continue;
    put(v_pool + at[r] * DV + c, f[r]);
    if (c < dk) *reinterpret_cast<uint4*>(k_pool + at[r] * dk + c) = key[r];
    for (int i = c + DV; i < dk; i += DV)
      *reinterpret_cast<uint4*>(k_pool + at[r] * dk + i) = *reinterpret_cast<const uint4*>(k + tok[r] * k_stride + g[r] * dk + i);
  }
}

// ---- RMS norm of a recurrence's fp32 read-outs [tokens, H, dv] -> T, with a weight, a gate and a factor as the mixer has them ----------
// Bound by bytes and, with a gate, nearly as much by the instructions of its sigmoids.  LPR lanes per row, eight elements per lane and
// piece; the rows of kHeadRows passes are under way before the first is waited for, and a row's token and head are counted on from the
// warp's first row (a division per row of four elements per lane was a sixth of the instructions).
// B200, bf16, 16384 x 8 rows of 128 with a gate: 52 -> 32 us (sigmoids one by one 34; copying as many bytes: 29); without one 29 -> 27.
constexpr int kHeadRows = 2;

struct HeadNorm {
  void* out; int64_t out_stride;           // per token
  const float* x;
  const void* w;                           // [dv] or null
  const void* gate; int64_t gate_stride;   // per token, or null
  int act;                                 // 0: sigmoid(g), 1: g sigmoid(g)
  float out_scale, eps;
  int64_t rows;
  int H, dv;
};

template <typename T>
struct alignas(16) Eight {
  T e[8];
};

template <typename T, int LPR, int NCH>
__global__ void __launch_bounds__(256)
head_norm_rows(const HeadNorm A) {
  constexpr int kPass = 32 / LPR;                      // rows of a warp at once
  const int64_t row0 = (static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5)) * (kHeadRows * kPass) + (threadIdx.x & 31) / LPR;
  const int c0 = (threadIdx.x % LPR) * 8, dv = A.dv;
  float v[kHeadRows][NCH][8];
  Eight<T> g[kHeadRows][NCH];
  int64_t at[kHeadRows];                               // token
  int h[kHeadRows];
  at[0] = static_cast<uint32_t>(row0) / static_cast<uint32_t>(A.H);
  h[0] = static_cast<int>(row0 - at[0] * A.H);
#pragma unroll
  for (int r = 0; r < kHeadRows; ++r) {
    if (r > 0) {
      at[r] = at[r - 1], h[r] = h[r - 1] + kPass;
      while (h[r] >= A.H) h[r] -= A.H, ++at[r];
    }
    const int64_t row = row0 + r * kPass;
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const int c = c0 + 8 * LPR * j;
      if (row < A.rows && c < dv) {
        get(v[r][j], A.x + row * dv + c);
        if (A.gate) g[r][j] = *reinterpret_cast<const Eight<T>*>(static_cast<const T*>(A.gate) + at[r] * A.gate_stride + h[r] * dv + c);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) v[r][j][u] = 0.f;
      }
    }
  }
  Eight<T> w[NCH];
#pragma unroll
  for (int j = 0; j < NCH; ++j)
    if (A.w && c0 + 8 * LPR * j < dv) w[j] = *reinterpret_cast<const Eight<T>*>(static_cast<const T*>(A.w) + c0 + 8 * LPR * j);
#pragma unroll
  for (int r = 0; r < kHeadRows; ++r) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NCH; ++j) ss += squares(v[r][j]);
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (row0 + r * kPass >= A.rows) continue;
    const float inv = rsqrtf(ss / static_cast<float>(dv) + A.eps);
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const int c = c0 + 8 * LPR * j;
      if (c >= dv) continue;
#pragma unroll
      for (int u = 0; u < 8; u += 2) {
        float y0 = v[r][j][u] * inv, y1 = v[r][j][u + 1] * inv;
        if (A.w) y0 *= Cvt<T>::to_f32(w[j].e[u]), y1 *= Cvt<T>::to_f32(w[j].e[u + 1]);
        if (A.gate) {
          const float z0 = Cvt<T>::to_f32(g[r][j].e[u]), z1 = Cvt<T>::to_f32(g[r][j].e[u + 1]);
          const float2 s = row_logistic2(z0, z1);
          y0 *= A.act == 1 ? z0 * s.x : s.x, y1 *= A.act == 1 ? z1 * s.y : s.y;
        }
        v[r][j][u] = y0 * A.out_scale, v[r][j][u + 1] = y1 * A.out_scale;
      }
      put(static_cast<T*>(A.out) + at[r] * A.out_stride + h[r] * dv + c, v[r][j]);
    }
  }
}
// element-wise form
template <typename T>
__global__ void __launch_bounds__(256)
head_norm_kernel(const HeadNorm A) {
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= A.rows) return;
  const int lane = threadIdx.x & 31, dv = A.dv;
  const float* xr = A.x + row * dv;
  float ss = 0.f;
  for (int i = lane; i < dv; i += 32) ss = fmaf(xr[i], xr[i], ss);
  const float inv = rsqrtf(warp_sum(ss) / static_cast<float>(dv) + A.eps);
  const int64_t n = row / A.H;
  const int h = static_cast<int>(row - n * A.H);
  const T* w = static_cast<const T*>(A.w);
  const T* gr = A.gate ? static_cast<const T*>(A.gate) + n * A.gate_stride + static_cast<int64_t>(h) * dv : nullptr;
  T* orow = static_cast<T*>(A.out) + n * A.out_stride + static_cast<int64_t>(h) * dv;
  for (int i = lane; i < dv; i += 32) {
    float y = xr[i] * inv;
    if (w) y *= Cvt<T>::to_f32(w[i]);
    if (gr) {
      const float g = Cvt<T>::to_f32(gr[i]);
      y *= A.act == 1 ? g * row_logistic(g) : row_logistic(g);
    }
    orow[i] = Cvt<T>::from_f32(y * A.out_scale);
  }
}

// ---- PolyNorm ---------------------------------------------------------------------------------------------------
template <typename T, int WPR, int NCH>
__global__ void __launch_bounds__(RowCta<WPR>::kNT)
polynorm_rows(T* __restrict__ out, const T* __restrict__ z, int64_t z_stride, const T* __restrict__ coef, float eps, int64_t rows, int ff) {
  __shared__ float red[24];
  const int64_t row = my_row<WPR>();
  if (row >= rows) return;
  float a[NCH][8], s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < ff) {
      get(a[c], z + row * z_stride + i);
      float a2[8], a3[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        a2[u] = a[c][u] * a[c][u];
        a3[u] = a2[u] * a[c][u];
      }
      s1 += squares(a[c]);
      s2 += squares(a2);
      s3 += squares(a3);
    }
  }
  const float n = static_cast<float>(ff);
  const float i1 = rsqrtf(row_sum<WPR>(s1, red) / n + eps);
  const float i2 = rsqrtf(row_sum<WPR>(s2, red + 8) / n + eps);
  const float i3 = rsqrtf(row_sum<WPR>(s3, red + 16) / n + eps);
  const float ca = Cvt<T>::to_f32(coef[0]), cb = Cvt<T>::to_f32(coef[1]), cc = Cvt<T>::to_f32(coef[2]), ce = Cvt<T>::to_f32(coef[3]);
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = my_piece<WPR>(c);
    if (i < ff) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float a1 = a[c][u], a2 = a1 * a1;
        a[c][u] = ca * a1 * i1 + cb * a2 * i2 + cc * a2 * a1 * i3 + ce;
      }
      put(out + row * ff + i, a[c]);
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(256)
polynorm_kernel(T* __restrict__ out, const T* __restrict__ z, int64_t z_stride, const T* __restrict__ coef, float eps,
                int ff) {
  __shared__ float red[32];
  const T* zr = z + static_cast<int64_t>(blockIdx.x) * z_stride;
  float s1 = 0.f, s2 = 0.f, s3 = 0.f;
  for (int i = threadIdx.x; i < ff; i += blockDim.x) {
    const float a = Cvt<T>::to_f32(zr[i]);
    const float a2 = a * a, a3 = a2 * a;
    s1 = fmaf(a, a, s1);
    s2 = fmaf(a2, a2, s2);
    s3 = fmaf(a3, a3, s3);
  }
  const float n = static_cast<float>(ff);
  const float i1 = rsqrtf(block_sum(s1, red) / n + eps);
  const float i2 = rsqrtf(block_sum(s2, red) / n + eps);
  const float i3 = rsqrtf(block_sum(s3, red) / n + eps);
  const float ca = Cvt<T>::to_f32(coef[0]), cb = Cvt<T>::to_f32(coef[1]), cc = Cvt<T>::to_f32(coef[2]),
              ce = Cvt<T>::to_f32(coef[3]);
  T* orow = out + static_cast<int64_t>(blockIdx.x) * ff;
  for (int i = threadIdx.x; i < ff; i += blockDim.x) {
    const float a = Cvt<T>::to_f32(zr[i]);
    const float a2 = a * a;
    orow[i] = Cvt<T>::from_f32(ca * a * i1 + cb * a2 * i2 + cc * a2 * a * i3 + ce);
  }
}

// ---- blocks of several pools set to zero (the pages of a finished request, all layers in one launch) -------------------
// The slots travel as a kernel argument: no copy to the device and nothing to keep until it has run.
constexpr int kZeroPools = 32, kZeroSlots = 640;
struct ZeroBlocks {
  char* pool[kZeroPools];
  int64_t bytes[kZeroPools];     // of a block, a multiple of 16
  int32_t slot[kZeroSlots];
};
__global__ void __launch_bounds__(256) zero_blocks_kernel(const __grid_constant__ ZeroBlocks A) {
  const int64_t n = A.bytes[blockIdx.y];
  uint4* dst = reinterpret_cast<uint4*>(A.pool[blockIdx.y] + A.slot[blockIdx.x] * n);
  for (int64_t i = threadIdx.x; i < n / 16; i += blockDim.x) dst[i] = make_uint4(0, 0, 0, 0);
}

// ---- expert order -------------------------------------------------------------------------------------------------
// One CTA of 32 warps; a warp owns the pairs of a contiguous chunk, 32 at a time, and keeps its ids in registers.  A pair's place among those of
// its expert in the chunk is what the chunk's earlier rounds left plus the lanes in front with the same id; an expert's counts are then summed
// over the chunks (a warp per expert): a stable counting sort.  Ids outside 0 .. E - 1 sort behind the last expert, so that order and where
// are permutations whatever the ids are: they index rows in the kernels that follow.
// B200, 8 experts: 8198 pairs 8.1 us (a chunk of ids per thread, read one after the other: 12.9; a radix sort of the same pairs is eight launches, 49).
constexpr int kOrderNT = 1024, kOrderWarps = kOrderNT / 32;
constexpr int kOrderExperts = 48, kOrderPairs = 16384;
__global__ void __launch_bounds__(kOrderNT)
expert_order_kernel(int64_t* __restrict__ order, int64_t* __restrict__ where, int32_t* __restrict__ offsets, const int32_t* __restrict__ ids,
                    int n_pairs, int E) {
  constexpr int kRounds = kOrderPairs / kOrderNT;
  __shared__ int count[kOrderExperts + 1][kOrderWarps + 1];     // (the last for ids of no expert)
  __shared__ int start[kOrderExperts + 2];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int rounds = (n_pairs + kOrderNT - 1) / kOrderNT, first = warp * rounds * 32 + lane;
  int bin[kRounds], rank[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int i = first + 32 * r;
    bin[r] = r < rounds && i < n_pairs ? static_cast<int>(min(static_cast<unsigned>(ids[i]), static_cast<unsigned>(E))) : -1;
  }
  for (int e = lane; e <= E; e += 32) count[e][warp] = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    if (r >= rounds) break;
    const unsigned same = __match_any_sync(0xffffffffu, bin[r]);
    const int before = __popc(same & ((1u << lane) - 1));
    int had = 0;
    if (bin[r] >= 0) had = count[bin[r]][warp];
    __syncwarp();
    if (bin[r] >= 0 && before == 0) count[bin[r]][warp] = had + __popc(same);
    __syncwarp();
    rank[r] = had + before;
  }
  __syncthreads();
  for (int e = warp; e <= E; e += kOrderWarps) {        // lane = chunk
    const int v = count[e][lane];
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    count[e][lane] = s - v;
    if (lane == 31) start[e + 1] = s;
  }
  __syncthreads();
  if (t == 0) {
    start[0] = 0;
    for (int e = 0; e <= E; ++e) start[e + 1] += start[e];
  }
  __syncthreads();
  if (t <= E) offsets[t] = start[t];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    if (bin[r] < 0) continue;
    const int i = first + 32 * r, at = start[bin[r]] + count[bin[r]][warp] + rank[r];
    order[at] = i;
    where[i] = at;
  }
}

// ---- rows of the expert-sorted input: xs[r] = T(w[src[r]] * h[src[r] / top]) ------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(128)
scaled_gather_kernel(T* __restrict__ xs, const T* __restrict__ h, const float* __restrict__ weights,
                     const int64_t* __restrict__ src, int top, int width) {
  const int64_t pair = src[blockIdx.x];
  const float w = weights[pair];
  const T* hr = h + (pair / top) * width;
  T* o = xs + static_cast<int64_t>(blockIdx.x) * width;
  for (int i = threadIdx.x * N; i < width; i += 128 * N) {
    if constexpr (N == 1) {
      o[i] = Cvt<T>::from_f32(w * Cvt<T>::to_f32(hr[i]));
    } else {
      float f[N];
      get(f, hr + i);
#pragma unroll
      for (int u = 0; u < N; ++u) f[u] *= w;
      put(o + i, f);
    }
  }
}

// ---- y = g' * sigmoid(alpha g') * (u' + 1), g' = min(g, limit), u' = clamp(u, -limit, limit); gu rows hold g | u ---------
template <typename T, int N>
__global__ void __launch_bounds__(256)
clamped_glu_kernel(T* __restrict__ y, const T* __restrict__ gu, int64_t rows, int ff, float limit, float alpha) {
  const int64_t n = rows * (ff / N);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / (ff / N);
    const int c = static_cast<int>(i - r * (ff / N)) * N;
    float a[N], b[N];
    if constexpr (N == 1) {
      a[0] = Cvt<T>::to_f32(gu[r * 2 * ff + c]);
      b[0] = Cvt<T>::to_f32(gu[r * 2 * ff + ff + c]);
    } else {
      get(a, gu + r * 2 * ff + c);
      get(b, gu + r * 2 * ff + ff + c);
    }
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const float g = fminf(a[u], limit);
      const float up = fminf(fmaxf(b[u], -limit), limit);
      a[u] = g * row_logistic(alpha * g) * (up + 1.0f);
    }
    if constexpr (N == 1) y[i] = Cvt<T>::from_f32(a[0]);
    else put(y + r * ff + c, a);
  }
}

// ---- out[n] = sum_k ys[where[n * top + k]] in fp32, k ascending ---------------------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(128)
expert_combine_kernel(float* __restrict__ out, const T* __restrict__ ys, const int64_t* __restrict__ where, int top,
                      int width) {
  const int64_t n = blockIdx.x;
  for (int i = threadIdx.x * N; i < width; i += 128 * N) {
    float a[N];
#pragma unroll
    for (int u = 0; u < N; ++u) a[u] = 0.f;
    for (int k = 0; k < top; ++k) {
      const T* src = ys + where[n * top + k] * width + i;
      if constexpr (N == 1) {
        a[0] += Cvt<T>::to_f32(src[0]);
      } else {
        float f[N];
        get(f, src);
#pragma unroll
        for (int u = 0; u < N; ++u) a[u] += f[u];
      }
    }
    if constexpr (N == 1) out[n * width + i] = a[0];
    else put(out + n * width + i, a);
  }
}

template <typename... P>
bool all16(const P*... p) {
  return (... && (p == nullptr || aligned16(p)));
}

// Rows in pieces of eight where every row of x, the gate and the output starts on a 16-byte boundary; dv beyond 512 would not stay in
// registers.
int head_norm(const HeadNorm& A, int dtype, void* stream, const char* name) {
  const auto s = static_cast<cudaStream_t>(stream);
  const bool whole = A.dv % 8 == 0 && A.dv <= 512 && A.out_stride % 8 == 0 && A.gate_stride % 8 == 0 && A.rows <= INT32_MAX &&
                     all16(A.out, A.x, A.w, A.gate);
  return rows_by_dtype(dtype, name, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto rows = [&](auto lpr, auto nch) {
      constexpr int LPR = decltype(lpr)::value, kPerCta = 8 * kHeadRows * 32 / LPR;
      head_norm_rows<T, LPR, decltype(nch)::value><<<static_cast<unsigned>((A.rows + kPerCta - 1) / kPerCta), 256, 0, s>>>(A);
    };
    using std::integral_constant;
    if (whole && A.dv <= 64) rows(integral_constant<int, 8>{}, integral_constant<int, 1>{});
    else if (whole && A.dv <= 128) rows(integral_constant<int, 16>{}, integral_constant<int, 1>{});
    else if (whole && A.dv <= 256) rows(integral_constant<int, 32>{}, integral_constant<int, 1>{});
    else if (whole) rows(integral_constant<int, 32>{}, integral_constant<int, 2>{});
    else head_norm_kernel<T><<<static_cast<unsigned>((A.rows + 7) / 8), 256, 0, s>>>(A);
    return check_launch(name);
  });
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int b200_offset_rmsnorm(void* out, const float* x, const void* weight, float eps, int rows, int width, int dtype,
                        void* stream) {
  if (rows < 0 || width <= 0) return fail(B200_EINVAL, "b200_offset_rmsnorm: bad sizes");
  if (rows == 0) return 0;
  if (!out || !x || !weight) return fail(B200_EINVAL, "b200_offset_rmsnorm: null pointer");
  const auto s = static_cast<cudaStream_t>(stream);
  return rows_by_dtype(dtype, "b200_offset_rmsnorm", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const bool whole = width % 8 == 0 && all16(out, x, weight) && by_row_shape(width, [&](auto wpr, auto nch) {
      constexpr int W = decltype(wpr)::value;
      offset_rmsnorm_rows<T, W, decltype(nch)::value><<<RowCta<W>::grid(rows), RowCta<W>::kNT, 0, s>>>(
          static_cast<T*>(out), x, static_cast<const T*>(weight), eps, rows, width);
    });
    if (!whole)
      offset_rmsnorm_kernel<T><<<rows, 256, 0, s>>>(static_cast<T*>(out), x, static_cast<const T*>(weight), eps, width);
    return check_launch("b200_offset_rmsnorm");
  });
}

int b200_postnorm_residual(float* x, const void* y, int64_t y_stride, int y_is_f32, const void* w_post, float mult,
                           const void* w_next, void* out_next, float eps, int rows, int width, int dtype, void* stream) {
  if (rows < 0 || width <= 0 || width > 40000) return fail(B200_EINVAL, "b200_postnorm_residual: bad sizes");
  if (rows == 0) return 0;
  if (!x || !y || !w_post || (w_next && !out_next)) return fail(B200_EINVAL, "b200_postnorm_residual: null pointer");
  const size_t smem = static_cast<size_t>(width) * sizeof(float);
  const auto s = static_cast<cudaStream_t>(stream);
  return rows_by_dtype(dtype, "b200_postnorm_residual", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto launch = [&](auto* ytag) {
      using Y = std::remove_pointer_t<decltype(ytag)>;
      const bool whole = width % 8 == 0 && y_stride % 8 == 0 && all16(x, y, w_post, w_next, out_next) &&
                         by_row_shape(width, [&](auto wpr, auto nch) {
        constexpr int W = decltype(wpr)::value;
        postnorm_residual_rows<T, Y, W, decltype(nch)::value><<<RowCta<W>::grid(rows), RowCta<W>::kNT, 0, s>>>(
            x, static_cast<const Y*>(y), y_stride, static_cast<const T*>(w_post), mult, static_cast<const T*>(w_next),
            static_cast<T*>(out_next), eps, rows, width);
      });
      if (whole) return;
      auto kern = postnorm_residual_kernel<T, Y>;
      if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
      kern<<<rows, 256, smem, s>>>(x, static_cast<const Y*>(y), y_stride, static_cast<const T*>(w_post), mult,
                                   static_cast<const T*>(w_next), static_cast<T*>(out_next), eps, width);
    };
    if (y_is_f32) launch(static_cast<float*>(nullptr));
    else launch(static_cast<T*>(nullptr));
    return check_launch("b200_postnorm_residual");
  });
}

int b200_value_prep_append(const void* k, int64_t k_stride, const void* v, int64_t v_stride, const void* v_prev,
                           void* v_keep, float lam, float eps, void* k_pool, void* v_pool, const int64_t* slot_mapping,
                           int n_tok, int G, int dk, int dv, int block_size, int64_t max_blocks, int dtype, void* stream) {
  if (n_tok < 0 || G <= 0 || dk <= 0 || dv <= 0 || block_size <= 0) return fail(B200_EINVAL, "b200_value_prep_append: bad sizes");
  if (n_tok == 0) return 0;
  if (!k || !v || !k_pool || !v_pool || !slot_mapping) return fail(B200_EINVAL, "b200_value_prep_append: null pointer");
  const int es = dtype_size(dtype);       // 0: refused below
  const bool four = es && dk % 4 == 0 && dv % 4 == 0 && k_stride % 4 == 0 && v_stride % 4 == 0 && all16(v_prev, v_keep, k_pool, v_pool) &&
                    reinterpret_cast<uintptr_t>(k) % (4 * es) == 0 && reinterpret_cast<uintptr_t>(v) % (4 * es) == 0;
  const unsigned grid = static_cast<unsigned>((static_cast<int64_t>(n_tok) * G + 7) / 8);
  return rows_by_dtype(dtype, "b200_value_prep_append", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto launch = [&](auto kern) {
      kern<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
          static_cast<const T*>(k), k_stride, static_cast<const T*>(v), v_stride, static_cast<const T*>(v_prev),
          static_cast<T*>(v_keep), lam, eps, static_cast<T*>(k_pool), static_cast<T*>(v_pool), slot_mapping, n_tok, G, dk, dv,
          block_size, max_blocks);
    };
    if constexpr (sizeof(T) == 2) {
      const int64_t rows = static_cast<int64_t>(n_tok) * G;
      auto pieces = [&](auto lpr) {
        constexpr int LPR = decltype(lpr)::value, kPerCta = 8 * kPrepRows * 32 / LPR;
        value_prep_rows<T, LPR><<<static_cast<unsigned>((rows + kPerCta - 1) / kPerCta), 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const T*>(k), k_stride, static_cast<const T*>(v), v_stride, static_cast<const T*>(v_prev), static_cast<T*>(v_keep), lam,
            eps, static_cast<T*>(k_pool), static_cast<T*>(v_pool), slot_mapping, rows, G, dk, block_size, max_blocks);
        return check_launch("b200_value_prep_append");
      };
      if (dk % 8 == 0 && k_stride % 8 == 0 && v_stride % 8 == 0 && all16(k, v, v_prev, v_keep, k_pool, v_pool) && rows <= INT32_MAX) {
        if (dv == 64) return pieces(std::integral_constant<int, 8>{});
        if (dv == 128) return pieces(std::integral_constant<int, 16>{});
        if (dv == 256) return pieces(std::integral_constant<int, 32>{});
      }
    }
    if (four) launch(value_prep_append_kernel<T, 4>);
    else launch(value_prep_append_kernel<T, 1>);
    return check_launch("b200_value_prep_append");
  });
}

int b200_head_rmsnorm(void* out, const float* x, const void* weight, float eps, int64_t rows, int dv, int dtype,
                      void* stream) {
  if (rows < 0 || dv <= 0) return fail(B200_EINVAL, "b200_head_rmsnorm: bad sizes");
  if (rows == 0) return 0;
  if (!out || !x || !weight) return fail(B200_EINVAL, "b200_head_rmsnorm: null pointer");
  return head_norm(HeadNorm{out, dv, x, weight, nullptr, 0, 0, 1.0f, eps, rows, 1, dv}, dtype, stream, "b200_head_rmsnorm");
}

int b200_head_rmsnorm_gated(void* out, const float* x, const void* weight, const void* gate, int64_t gate_stride, float eps,
                            int64_t n_tok, int H, int dv, int dtype, void* stream) {
  if (n_tok < 0 || H <= 0 || dv <= 0) return fail(B200_EINVAL, "b200_head_rmsnorm_gated: bad sizes");
  if (n_tok == 0) return 0;
  if (!out || !x || !weight) return fail(B200_EINVAL, "b200_head_rmsnorm_gated: null pointer");
  return head_norm(HeadNorm{out, static_cast<int64_t>(H) * dv, x, weight, gate, gate_stride, 0, 1.0f, eps, n_tok * H, H, dv}, dtype, stream,
                   "b200_head_rmsnorm_gated");
}

int b200_head_norm_act_gate(void* out, int64_t out_stride, const float* x, const void* weight, const void* gate,
                            int64_t gate_stride, int gate_act, float out_scale, float eps, int64_t n_tok, int H, int dv,
                            int dtype, void* stream) {
  if (n_tok < 0 || H <= 0 || dv <= 0 || gate_act < 0 || gate_act > 1)
    return fail(B200_EINVAL, "b200_head_norm_act_gate: bad sizes");
  if (n_tok == 0) return 0;
  if (!out || !x) return fail(B200_EINVAL, "b200_head_norm_act_gate: null pointer");
  return head_norm(HeadNorm{out, out_stride, x, weight, gate, gate_stride, gate_act, out_scale, eps, n_tok * H, H, dv}, dtype, stream,
                   "b200_head_norm_act_gate");
}

int b200_polynorm(void* out, const void* z, int64_t z_stride, const void* coef, float eps, int rows, int ff, int dtype,
                  void* stream) {
  if (rows < 0 || ff <= 0) return fail(B200_EINVAL, "b200_polynorm: bad sizes");
  if (rows == 0) return 0;
  if (!out || !z || !coef) return fail(B200_EINVAL, "b200_polynorm: null pointer");
  const auto s = static_cast<cudaStream_t>(stream);
  return rows_by_dtype(dtype, "b200_polynorm", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const bool whole = ff % 8 == 0 && z_stride % 8 == 0 && all16(out, z) && by_row_shape(ff, [&](auto wpr, auto nch) {
      constexpr int W = decltype(wpr)::value;
      polynorm_rows<T, W, decltype(nch)::value><<<RowCta<W>::grid(rows), RowCta<W>::kNT, 0, s>>>(
          static_cast<T*>(out), static_cast<const T*>(z), z_stride, static_cast<const T*>(coef), eps, rows, ff);
    });
    if (!whole)
      polynorm_kernel<T><<<rows, 256, 0, s>>>(static_cast<T*>(out), static_cast<const T*>(z), z_stride, static_cast<const T*>(coef), eps, ff);
    return check_launch("b200_polynorm");
  });
}

int b200_zero_blocks(void* const* pools, const int64_t* block_bytes, int n_pools, const int32_t* slots, int n_slots, void* stream) {
  if (n_pools < 0 || n_slots < 0) return fail(B200_EINVAL, "b200_zero_blocks: bad sizes");
  if (n_pools == 0 || n_slots == 0) return 0;
  if (!pools || !block_bytes || !slots) return fail(B200_EINVAL, "b200_zero_blocks: null pointer");
  for (int p0 = 0; p0 < n_pools; p0 += kZeroPools) {
    ZeroBlocks A{};
    const int np = std::min(kZeroPools, n_pools - p0);
    for (int i = 0; i < np; ++i) {
      A.pool[i] = static_cast<char*>(pools[p0 + i]);
      A.bytes[i] = block_bytes[p0 + i];
      if (!A.pool[i] || !aligned16(A.pool[i]) || A.bytes[i] < 0 || A.bytes[i] % 16)
        return fail(B200_ESHAPE, "b200_zero_blocks: blocks are whole 16-byte words");
    }
    for (int s0 = 0; s0 < n_slots; s0 += kZeroSlots) {
      const int ns = std::min(kZeroSlots, n_slots - s0);
      for (int i = 0; i < ns; ++i) A.slot[i] = slots[s0 + i];
      zero_blocks_kernel<<<dim3(ns, np), 256, 0, static_cast<cudaStream_t>(stream)>>>(A);
    }
  }
  return check_launch("b200_zero_blocks");
}

int b200_expert_order_supported(int64_t n_pairs, int n_experts) {
  return n_pairs >= 0 && n_pairs <= kOrderPairs && n_experts > 0 && n_experts <= kOrderExperts;
}

int b200_expert_order(int64_t* order, int64_t* where, int32_t* offsets, const int32_t* ids, int64_t n_pairs, int n_experts, void* stream) {
  if (!b200_expert_order_supported(n_pairs, n_experts)) return fail(B200_ESHAPE, "b200_expert_order: up to %d pairs and %d experts", kOrderPairs, kOrderExperts);
  if (!offsets || (n_pairs > 0 && (!order || !where || !ids))) return fail(B200_EINVAL, "b200_expert_order: null pointer");
  expert_order_kernel<<<1, kOrderNT, 0, static_cast<cudaStream_t>(stream)>>>(order, where, offsets, ids, static_cast<int>(n_pairs), n_experts);
  return check_launch("b200_expert_order");
}

int b200_scaled_gather(void* xs, const void* h, const float* weights, const int64_t* src, int64_t n_rows, int top,
                       int width, int dtype, void* stream) {
  if (n_rows < 0 || top <= 0 || width <= 0) return fail(B200_EINVAL, "b200_scaled_gather: bad sizes");
  if (n_rows == 0) return 0;
  if (!xs || !h || !weights || !src) return fail(B200_EINVAL, "b200_scaled_gather: null pointer");
  return rows_by_dtype(dtype, "b200_scaled_gather", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto launch = [&](auto kern) {
      kern<<<static_cast<unsigned>(n_rows), 128, 0, static_cast<cudaStream_t>(stream)>>>(
          static_cast<T*>(xs), static_cast<const T*>(h), weights, src, top, width);
    };
    if (width % 8 == 0 && all16(xs, h)) launch(scaled_gather_kernel<T, 8>);
    else launch(scaled_gather_kernel<T, 1>);
    return check_launch("b200_scaled_gather");
  });
}

int b200_clamped_glu(void* y, const void* gu, int64_t rows, int ff, float limit, float alpha, int dtype, void* stream) {
  if (rows < 0 || ff <= 0) return fail(B200_EINVAL, "b200_clamped_glu: bad sizes");
  if (rows == 0) return 0;
  if (!y || !gu) return fail(B200_EINVAL, "b200_clamped_glu: null pointer");
  const bool eight = ff % 8 == 0 && all16(y, gu);
  const int64_t n = rows * ff / (eight ? 8 : 1);
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, kNumSMs * 16));
  return rows_by_dtype(dtype, "b200_clamped_glu", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto launch = [&](auto kern) {
      kern<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<T*>(y), static_cast<const T*>(gu), rows, ff, limit, alpha);
    };
    if (eight) launch(clamped_glu_kernel<T, 8>);
    else launch(clamped_glu_kernel<T, 1>);
    return check_launch("b200_clamped_glu");
  });
}

int b200_expert_combine(float* out, const void* ys, const int64_t* where, int64_t n_tok, int top, int width, int dtype,
                        void* stream) {
  if (n_tok < 0 || top <= 0 || width <= 0) return fail(B200_EINVAL, "b200_expert_combine: bad sizes");
  if (n_tok == 0) return 0;
  if (!out || !ys || !where) return fail(B200_EINVAL, "b200_expert_combine: null pointer");
  return rows_by_dtype(dtype, "b200_expert_combine", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto launch = [&](auto kern) {
      kern<<<static_cast<unsigned>(n_tok), 128, 0, static_cast<cudaStream_t>(stream)>>>(out, static_cast<const T*>(ys), where, top, width);
    };
    if (width % 8 == 0 && all16(out, ys)) launch(expert_combine_kernel<T, 8>);
    else launch(expert_combine_kernel<T, 1>);
    return check_launch("b200_expert_combine");
  });
}

}  // extern "C"
