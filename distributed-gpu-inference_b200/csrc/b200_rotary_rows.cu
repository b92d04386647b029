// Rows with rotary positions on their way into the pages, 16-bit types, in 16-byte pieces: per-head norms of q and k, rotation, append
// (b200_parallel_ops.cu has the element-wise form), and the latent rows of absorbed attention (b200_gated_ops.cu).
//
// What bounds them: the element-wise kernels had one CTA per token, whose angles (double precision, as many threads busy as there are
// frequencies) and rows came one after the other: 3300 tokens of 16 + 4 heads of 128 took 29.6 us, a fifth of what their bytes would allow.
// Here the angles of a CTA's tokens fill its threads, the first rows are asked for before the angles are computed, a lane moves eight
// elements, a row's sum of squares and the partners of its rotation are a few shuffles among its 8, 16 or 32 lanes.
// B200, bf16, before -> now: q and k of 16 + 4 heads of 128, 64 turned: 1 token 3.3 -> 3.2 us, 591: 7.3 -> 4.7, 3300: 29.6 -> 13.0,
// 16384: 158 -> 55 (201 MB); latent rows of 256 + 64 with 16 query parts of 64: 1 token 3.3 -> 2.9, 591: 6.2 -> 3.6, 3300: 15.1 -> 6.6,
// 16384: 65 -> 28 (88 MB).
#include <type_traits>

#include "b200_common.cuh"
#include "b200_rotary_rows.cuh"

namespace b200 {
namespace {

constexpr int kNT = 256, kWarps = kNT / 32, kMaxToks = kWarps;
constexpr int kWave = 4 * 148;      // CTAs at once: 62 registers a thread

// Tokens per CTA: as few as keep the grid within one wave, up to eight.  us for 1 / 2 / 4 / 8 tokens each, q and k of 16 + 4 heads of 128:
// 147 tokens 3.6 / 4.1 / 5.1 / -, 800: 7.2 / 5.3 / 6.1 / -, 2200: 13.7 / 10.9 / 9.3 / 10.2, 16384: 102 / 71 / 58 / 55.
int tokens_per_cta(int n_tok) {
  int per = 1;
  while (per < kMaxToks && n_tok > per * kWave) per *= 2;
  return per;
}

template <typename T>
union Piece {
  uint4 raw;
  T e[8];
};
template <typename T>
__device__ __forceinline__ Piece<T> piece(const T* p) {
  Piece<T> r;
  r.raw = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <typename T>
__device__ __forceinline__ void widen(float (&d)[8], const Piece<T>& p) {
#pragma unroll
  for (int i = 0; i < 8; ++i) d[i] = Cvt<T>::to_f32(p.e[i]);
}
template <typename T>
__device__ __forceinline__ void put(T* to, const float (&d)[8]) {
  Piece<T> p;
#pragma unroll
  for (int i = 0; i < 8; ++i) p.e[i] = Cvt<T>::from_f32(d[i]);
  *reinterpret_cast<uint4*>(to) = p.raw;
}

// (cos, sin) of the CTA's tokens and frequencies, times gain
__device__ __forceinline__ void angles(float2* cs, const int32_t* tok_pos, int tok0, int toks, const double* freqs, int half, float gain) {
  for (int i = threadIdx.x; i < toks * half; i += kNT) {
    const int t = i / half;
    double s, c;
    sincos(static_cast<double>(tok_pos[tok0 + t]) * freqs[i - t * half], &s, &c);
    cs[i] = make_float2(static_cast<float>(c) * gain, static_cast<float>(s) * gain);
  }
}

// LPR lanes per row of 8 LPR elements
template <typename T, int LPR>
__global__ void __launch_bounds__(kNT)
qk_rows_kernel(const QkRows A, int per) {
  extern __shared__ float2 cs[];      // [per][rot_dims / 2]
  constexpr int kRows = 32 / LPR, DK = 8 * LPR;
  const int tok0 = blockIdx.x * per, toks = min(per, A.n_tok - tok0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = lane % LPR, sub = lane / LPR;
  const int heads = A.H + A.G, items = toks * heads, half = A.rot_dims / 2, hp = half / 8;
  T* q = static_cast<T*>(A.q);
  const T* k = static_cast<const T*>(A.k);
  const int first = warp * kRows + sub;
  auto where = [&](int item, int& t, int& hh) {
    t = item / heads;
    hh = item - t * heads;
  };
  auto load = [&](int item) {
    int t, hh;
    where(min(item, items - 1), t, hh);
    const int64_t n = tok0 + t;
    return piece(hh < A.H ? q + n * A.q_stride + hh * DK + 8 * c : k + n * A.k_stride + (hh - A.H) * DK + 8 * c);
  };
  Piece<T> next = load(first), qw, kw;
  if (A.qw) qw = piece(static_cast<const T*>(A.qw) + 8 * c);
  if (A.kw) kw = piece(static_cast<const T*>(A.kw) + 8 * c);
  angles(cs, A.tok_pos, tok0, toks, A.freqs, half, 1.0f);
  __syncthreads();
  for (int item0 = warp * kRows; item0 < items; item0 += kWarps * kRows) {     // the same for a warp: its rows shuffle together
    const int item = item0 + sub;
    float x[8];
    widen(x, next);
    next = load(item + kWarps * kRows);
    int t, hh;
    where(min(item, items - 1), t, hh);
    const bool is_q = hh < A.H;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = fmaf(x[i], x[i], ss);
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const bool weight = is_q ? A.qw != nullptr : A.kw != nullptr;
    if (weight || A.unit_norm) {      // a rotation keeps the row's length: without a weight, before it is after it
      const float inv = rsqrtf(ss / static_cast<float>(DK) + A.eps);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = x[i] * inv * (weight ? Cvt<T>::to_f32(is_q ? qw.e[i] : kw.e[i]) : 1.0f);
    }
    const float2* at = cs + t * half;
    if (A.interleaved) {
      if (8 * c < A.rot_dims) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = at[4 * c + i];
          const float u = x[2 * i], w = x[2 * i + 1];
          x[2 * i] = u * a.x - w * a.y;
          x[2 * i + 1] = w * a.x + u * a.y;
        }
      }
    } else {
      const int pc = c < hp ? c + hp : c < 2 * hp ? c - hp : c;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float other = __shfl_sync(0xffffffffu, x[i], lane - c + pc);
        if (c < 2 * hp) {
          const float2 a = at[8 * (c < hp ? c : pc) + i];
          x[i] = c < hp ? x[i] * a.x - other * a.y : x[i] * a.x + other * a.y;
        }
      }
    }
    if (item >= items) continue;
    const int64_t n = tok0 + t;
    if (is_q) {
      put(q + n * A.q_stride + hh * DK + 8 * c, x);
    } else {
      const int64_t slot = A.slot_mapping[n];
      if (slot >= 0) {
        const int64_t blk = slot / A.block_size;
        put(static_cast<T*>(A.k_pool) + ((blk * A.G + hh - A.H) * A.block_size + (slot - blk * A.block_size)) * DK + 8 * c, x);
      }
    }
  }
  const int per_head = A.dv / 8, per_tok = A.Gv * per_head;
  for (int i = threadIdx.x; i < toks * per_tok; i += kNT) {
    const int t = i / per_tok, p = i - t * per_tok, g = p / per_head, at = p - g * per_head;
    const int64_t n = tok0 + t, slot = A.slot_mapping[n];
    if (slot < 0) continue;
    const int64_t blk = slot / A.block_size;
    *reinterpret_cast<uint4*>(static_cast<T*>(A.v_pool) + ((blk * A.Gv + g) * A.block_size + (slot - blk * A.block_size)) * A.dv + 8 * at) =
        piece(static_cast<const T*>(A.v) + n * A.v_stride + 8 * p).raw;
  }
}

template <typename T>
__global__ void __launch_bounds__(kNT)
latent_rows_kernel(const LatentRows A, int per) {
  extern __shared__ float2 cs[];
  const int tok0 = blockIdx.x * per, toks = min(per, A.n_tok - tok0), half = A.rot_dims / 2, hp = half / 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_head = A.dr / 8, items = toks * A.H * per_head;
  auto source = [&](int i, int& t, int& h, int& c) {
    const int row = i / per_head;
    c = i - row * per_head;
    t = row / A.H;
    h = row - t * A.H;
    return static_cast<const T*>(A.q) + static_cast<int64_t>(tok0 + t) * A.q_tok_stride + static_cast<int64_t>(h) * A.q_head_stride;
  };
  auto partner = [&](int c) { return c < hp ? c + hp : c - hp; };
  // x: piece c of a rotated part, other: its partner (c, -) where pairs are half the rotated dimensions apart
  auto turn = [&](float (&x)[8], const float (&other)[8], int t, int c) {
    const float2* at = cs + t * half;
    if (8 * c >= A.rot_dims) return;
    if (A.interleaved) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = at[4 * c + i];
        const float u = x[2 * i], v = x[2 * i + 1];
        x[2 * i] = fmaf(u, a.x, -v * a.y);
        x[2 * i + 1] = fmaf(v, a.x, u * a.y);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 a = at[8 * (c < hp ? c : c - hp) + i];
        x[i] = c < hp ? fmaf(x[i], a.x, -other[i] * a.y) : fmaf(x[i], a.x, other[i] * a.y);
      }
    }
  };
  auto rotated = [&](const T* part, int t, int c, T* to) {
    float x[8], other[8];
    widen(x, piece(part + 8 * c));
    if (!A.interleaved && 8 * c < A.rot_dims) widen(other, piece(part + 8 * partner(c)));
    turn(x, other, t, c);
    put(to, x);
  };
  // the latents: a warp per token
  const bool mine = warp < toks;
  const int64_t n = tok0 + (mine ? warp : 0), slot = A.slot_mapping[n];
  const T* row = static_cast<const T*>(A.dkv) + n * A.dkv_stride;
  T* dst = static_cast<T*>(A.pool) + (slot >= 0 ? slot : 0) * (A.rank + A.dr);
  if (mine && slot >= 0) {
    Piece<T> p0;
    if (8 * lane < A.rank) p0 = piece(row + 8 * lane);
    float ss = 0.f;
    for (int i = 8 * lane; i < A.rank; i += 256) {
      float x[8];
      widen(x, i == 8 * lane ? p0 : piece(row + i));
#pragma unroll
      for (int u = 0; u < 8; ++u) ss = fmaf(x[u], x[u], ss);
    }
    const float inv = rsqrtf(warp_sum(ss) / static_cast<float>(A.rank) + A.eps);
    for (int i = 8 * lane; i < A.rank; i += 256) {
      float x[8], w[8];
      widen(x, i == 8 * lane ? p0 : piece(row + i));
      widen(w, piece(static_cast<const T*>(A.w_c) + i));
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = x[u] * inv * w[u];
      put(dst + i, x);
    }
  }
  angles(cs, A.tok_pos, tok0, toks, A.freqs, half, A.gain);
  __syncthreads();
  if (mine && slot >= 0) {
    for (int c = lane; c < per_head; c += 32) rotated(row + A.rank, warp, c, dst + A.rank + 8 * c);
  }
#pragma unroll 2
  for (int i = threadIdx.x; i < items; i += kNT) {
    int t, h, c;
    const T* part = source(i, t, h, c);
    rotated(part, t, c, static_cast<T*>(A.q_out) + static_cast<int64_t>(tok0 + t) * A.qo_tok_stride + static_cast<int64_t>(h) * A.qo_head_stride + 8 * c);
  }
}

bool rotation_fits(int rot_dims, int interleaved) { return rot_dims % (interleaved ? 8 : 16) == 0 && rot_dims <= 1024; }
template <typename... I>
bool eights(I... n) {
  return (... && (n % 8 == 0));
}
template <typename... P>
bool all16(const P*... p) {
  return (... && aligned16(p));     // null is
}

}  // namespace

bool qk_rows(const QkRows& A, int dtype, cudaStream_t stream) {
  if ((dtype != B200_DTYPE_F16 && dtype != B200_DTYPE_BF16) || (A.dk != 64 && A.dk != 128 && A.dk != 256)) return false;
  if (!rotation_fits(A.rot_dims, A.interleaved) || !eights(A.q_stride, A.k_stride, A.v_stride, A.dv) || !all16(A.q, A.k, A.v, A.qw, A.kw, A.k_pool, A.v_pool))
    return false;
  const int per = tokens_per_cta(A.n_tok);
  const unsigned grid = static_cast<unsigned>((A.n_tok + per - 1) / per);
  const size_t smem = sizeof(float2) * per * (A.rot_dims / 2);
  auto go = [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if (A.dk == 64) qk_rows_kernel<T, 8><<<grid, kNT, smem, stream>>>(A, per);
    else if (A.dk == 128) qk_rows_kernel<T, 16><<<grid, kNT, smem, stream>>>(A, per);
    else qk_rows_kernel<T, 32><<<grid, kNT, smem, stream>>>(A, per);
  };
  if (dtype == B200_DTYPE_F16) go(static_cast<__half*>(nullptr));
  else go(static_cast<__nv_bfloat16*>(nullptr));
  return true;
}

bool latent_rows(const LatentRows& A, int dtype, cudaStream_t stream) {
  if (dtype != B200_DTYPE_F16 && dtype != B200_DTYPE_BF16) return false;
  if (A.dr <= 0 || !rotation_fits(A.rot_dims, A.interleaved) ||
      !eights(A.dr, A.rank, A.q_tok_stride, A.q_head_stride, A.qo_tok_stride, A.qo_head_stride, A.dkv_stride) || !all16(A.q, A.q_out, A.dkv, A.w_c, A.pool))
    return false;
  const int per = tokens_per_cta(A.n_tok);
  const unsigned grid = static_cast<unsigned>((A.n_tok + per - 1) / per);
  const size_t smem = sizeof(float2) * per * (A.rot_dims / 2);
  if (dtype == B200_DTYPE_F16) latent_rows_kernel<__half><<<grid, kNT, smem, stream>>>(A, per);
  else latent_rows_kernel<__nv_bfloat16><<<grid, kNT, smem, stream>>>(A, per);
  return true;
}

}  // namespace b200
