// The three recurrences that walk a portion token by token with an fp32 state [dk][dv] per (sequence, head):
//
//   gated      S <- f_i S + (1 - f_i) v          o = S^T q     f = l + (1 - l) sigmoid(z + b) per key channel, q = silu(z_q)
//   delta      S <- S + (g_i - 1) S;  u = beta (v - S^T k);  S <- S + k u;  o = S^T q     g a decay per key channel or per head
//   retention  S <- d S + (c k) v^T              o = S^T q     d fixed per head
//
// A value column's part of the state never meets another column's, so columns are independent and the time of a launch is the
// length of one column's chain times the work of a token.  What bounds it is how a token's q, k and decays reach the lanes: they
// are the same for all columns, and a shared-memory read delivers 128 bytes per clock and SM however many lanes ask for the same
// word.  So a lane owns a TILE of the state, DK / 8 rows of C columns, and a row's value once read serves C columns; eight lanes
// make a column, a warp 4 C columns.  The rows of a lane are 32 j + 4 r .. + 3: eight lanes read 128 contiguous bytes.  The
// arithmetic is packed pairs of rows (fma.rn.f32x2: half the issue slots, the same rate).  Four more warps of the CTA prepare the
// next eight tokens meanwhile (loads four stages ahead by cp.async; activations, decays, unit norms once per CTA), so the columns'
// warps carry the recurrence only; one barrier per eight tokens.  Read-outs are reduced over the eight lanes for eight (token,
// column) pairs at once: seven shuffles instead of three per pair.
//
// Measured on B200, bf16, 64 x 128 states, against four lanes per column that prepare their own inputs: delta, 8 x 2048 tokens of 8
// heads 2302 -> 469 us; gated, 6 portions of up to 1900 tokens of 16 heads 1228 -> 396 us; retention, 5 portions of up to 1024 tokens
// of 16 heads 474 -> 157 us.  A token of one warp per scheduler takes 250 - 470 clocks, of which the packed multiply-adds are 130 - 190:
// what is left is the latency of a token's dependent steps, and larger steps overlap the chains of several CTAs.
#include <type_traits>

#include "b200_column_scan.cuh"
#include "b200_common.cuh"

namespace b200 {
namespace {

enum Rule { kGated, kDelta, kRetention };

struct ColSeq {
  int tok0, count, slot, fresh;
};

struct ColArgs {
  float* o;
  ScanRows in;
  const void* beta; int64_t beta_stride;
  const void* a; int64_t a_stride;
  const void* bias;       // gated: f_bias, delta: dt_bias
  const void* rate;       // gated: lower, delta: a_log
  const float* decay;     // retention
  float* state;
  const ColSeq* seqs;
  int H, G, dk, dv;
  int per_channel;        // delta: a decay logit and a bias per key channel (1) or one per head (0)
  int vec_qk, vec_a, vec_v, vec_s;   // four elements of q / k, a, v, four state columns can be moved at once
  float unit_eps, scale;  // delta: q_scale; retention: k_scale
};

constexpr int kStage = 8;        // tokens per stage
constexpr int kColWarps = 4;     // warps that own columns; as many prepare
constexpr int kColNT = 64 * kColWarps;

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ float logistic(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float soft_plus(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

// N consecutive elements of a row, `left` of which exist, into shared memory: without a register in between where the caller
// knows them aligned, so that any number of them can be under way.
template <int N, typename T>
__device__ __forceinline__ void stage_n(T* dst, const T* src, int left, bool vec) {
  if constexpr (N * sizeof(T) >= 4) {
    if (vec && left >= N) {
      const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(src), "n"(static_cast<int>(N * sizeof(T))) : "memory");
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) dst[i] = i < left ? src[i] : Cvt<T>::from_f32(0.f);
}
template <typename T>
__device__ __forceinline__ void read4(float (&d)[4], const T* p) {
  alignas(16) T e[4];
  if constexpr (sizeof(T) == 2) {
    *reinterpret_cast<uint2*>(e) = *reinterpret_cast<const uint2*>(p);
  } else {
    *reinterpret_cast<uint4*>(e) = *reinterpret_cast<const uint4*>(p);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] = Cvt<T>::to_f32(e[i]);
}

template <int RULE, int DK, int C>
struct Stage {
  static constexpr int kSections = RULE == kRetention ? 2 : 3;   // q | k, or q | f | 1 - f, or q | k | g - 1
  static constexpr int kRow = kSections * DK;
  static constexpr int kCols = 4 * C * kColWarps;
  float rows[kStage][kRow];
  float v[kStage][kCols];
  float beta[kStage];
};

// What the preparing threads have under way: every thread reads back only what it asked for itself.
template <int RULE, typename T, int DK, int C>
struct Flight {
  static constexpr int kDepth = DK <= 128 ? 4 : 2;                // stages
  static constexpr int kSections = RULE == kDelta ? 3 : 2;
  T rows[kDepth][kStage][kSections * DK];
  T v[kDepth][kStage][Stage<RULE, DK, C>::kCols];
};

template <int RULE, typename T, int DK, int C>
constexpr size_t column_smem() {
  return 2 * sizeof(Stage<RULE, DK, C>) + sizeof(Flight<RULE, T, DK, C>);
}

template <int RULE, typename T, int DK, int C>
__global__ void __launch_bounds__(kColNT)
column_scan_kernel(const ColArgs A) {
  using S_t = Stage<RULE, DK, C>;
  extern __shared__ __align__(16) unsigned char stage_raw[];
  S_t* stage = reinterpret_cast<S_t*>(stage_raw);      // two of them, then the loads under way
  constexpr int kCols = S_t::kCols;
  const ColSeq sq = A.seqs[blockIdx.x];
  const int h = blockIdx.y, H = A.H, dk = A.dk, dv = A.dv;
  const int col_cta = blockIdx.z * kCols;
  const int warp = threadIdx.x >> 5;
  const int n_stages = (sq.count + kStage - 1) / kStage;

  if (warp >= kColWarps) {
    // ---- the warps that prepare: 16 threads per token of a stage, four elements of every 64 each -------------------------
    const int p = threadIdx.x - 32 * kColWarps;
    const int tt = p >> 4, e0 = (p & 15) * 4;
    constexpr int NJ = (DK + 63) / 64;
    const int gq = h / (H / A.G);
    const T* qp = static_cast<const T*>(A.in.q) + gq * dk;
    const T* kp = static_cast<const T*>(A.in.k) + gq * dk;
    const T* vp = static_cast<const T*>(A.in.v) + h * dv + col_cta;
    const T* ap = static_cast<const T*>(A.a) + (RULE == kDelta && A.per_channel ? h * dk : h);
    const T* bp = static_cast<const T*>(A.beta) + h;
    const T* bias = static_cast<const T*>(A.bias);
    const T* rate = static_cast<const T*>(A.rate);
    float a_rate = 0.f;
    if constexpr (RULE == kDelta) a_rate = expf(Cvt<T>::to_f32(rate[h]));
    // constants of this thread's channels, kept where they fit registers
    constexpr bool kKeep = RULE != kRetention && NJ <= 2;
    float cb[kKeep ? NJ : 1][4], cr[kKeep ? NJ : 1][4];
    auto constants = [&](int j, float (&b4)[4], float (&r4)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = e0 + 64 * j + i;
        b4[i] = r4[i] = 0.f;
        if (e >= dk) continue;
        if constexpr (RULE == kGated) {
          b4[i] = Cvt<T>::to_f32(bias[h * dk + e]);
          r4[i] = Cvt<T>::to_f32(rate[h * dk + e]);
        } else if constexpr (RULE == kDelta) {
          b4[i] = Cvt<T>::to_f32(bias[A.per_channel ? h * dk + e : h]);
        }
      }
    };
    if constexpr (kKeep) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) constants(j, cb[j], cr[j]);
    }
    auto& fl = *reinterpret_cast<Flight<RULE, T, DK, C>*>(stage + 2);
    constexpr int kDepth = Flight<RULE, T, DK, C>::kDepth;
    auto fetch = [&](int s) {
      const int t = s * kStage + tt, slot = s % kDepth;
      if (t < sq.count) {
        const int64_t tok = sq.tok0 + t;
        T* row = fl.rows[slot][tt];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int e = e0 + 64 * j;
          if (e < DK) {
            stage_n<4>(row + e, qp + tok * A.in.stride + e, dk - e, A.vec_qk);
            stage_n<4>(row + DK + e, kp + tok * A.in.stride + e, dk - e, A.vec_qk);
            if constexpr (RULE == kDelta) {
              if (A.per_channel) stage_n<4>(row + 2 * DK + e, ap + tok * A.a_stride + e, dk - e, A.vec_a);
            }
          }
        }
        const int c0 = (p & 15) * C;
        stage_n<C>(&fl.v[slot][tt][c0], vp + tok * A.in.stride + c0, dv - col_cta - c0, A.vec_v);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // single 16-bit elements cannot be copied that way: one stage ahead in registers
    T rb = Cvt<T>::from_f32(0.f), ra = rb;
    auto scalars = [&](int s) {
      if constexpr (RULE == kDelta) {
        const int t = s * kStage + tt;
        if (t < sq.count) {
          const int64_t tok = sq.tok0 + t;
          rb = bp[tok * A.beta_stride];
          if (!A.per_channel) ra = ap[tok * A.a_stride];
        }
      }
    };
    auto commit = [&](int s) {       // kDepth - 1 later groups may still be under way
      asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
      const bool live = s * kStage + tt < sq.count;     // the same for the 16 threads of a token
      const int slot = s % kDepth;
      S_t& st = stage[s & 1];
      float x[NJ][4], y[NJ][4];
      float sq2 = 0.f, sk2 = 0.f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int e = e0 + 64 * j;
        if (live && e < DK) {
          read4(x[j], fl.rows[slot][tt] + e);
          read4(y[j], fl.rows[slot][tt] + DK + e);
        }
      }
      if constexpr (RULE == kDelta) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          if (live && e0 + 64 * j < DK) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              sq2 = fmaf(x[j][i], x[j][i], sq2);
              sk2 = fmaf(y[j][i], y[j][i], sk2);
            }
          }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          sq2 += __shfl_xor_sync(0xffffffffu, sq2, o);
          sk2 += __shfl_xor_sync(0xffffffffu, sk2, o);
        }
        sq2 = rsqrtf(sq2 + A.unit_eps) * A.scale;
        sk2 = rsqrtf(sk2 + A.unit_eps);
      }
      if (!live) return;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int e = e0 + 64 * j;
        if (e >= DK) continue;
        float z[4], b4[4], r4[4];
        if constexpr (kKeep) {
#pragma unroll
          for (int i = 0; i < 4; ++i) b4[i] = cb[j][i], r4[i] = cr[j][i];
        } else {
          constants(j, b4, r4);
        }
        if constexpr (RULE == kDelta) {
          if (A.per_channel) {
            read4(z, fl.rows[slot][tt] + 2 * DK + e);
          } else {
            z[0] = z[1] = z[2] = z[3] = Cvt<T>::to_f32(ra);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if constexpr (RULE == kGated) {
            // padded rows: q = f = 1 - f = 0, the state there stays 0
            const float f = r4[i] + (1.0f - r4[i]) * logistic(y[j][i] + b4[i]);
            x[j][i] = x[j][i] * logistic(x[j][i]);
            y[j][i] = e + i < dk ? f : 0.f;
            z[i] = e + i < dk ? 1.0f - f : 0.f;
          } else if constexpr (RULE == kDelta) {
            x[j][i] *= sq2;
            y[j][i] *= sk2;
            z[i] = e + i < dk ? expm1f(-a_rate * soft_plus(z[i] + b4[i])) : 0.f;
          } else {
            y[j][i] *= A.scale;
          }
        }
        *reinterpret_cast<float4*>(&st.rows[tt][e]) = make_float4(x[j][0], x[j][1], x[j][2], x[j][3]);
        *reinterpret_cast<float4*>(&st.rows[tt][DK + e]) = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
        if constexpr (RULE != kRetention) *reinterpret_cast<float4*>(&st.rows[tt][2 * DK + e]) = make_float4(z[0], z[1], z[2], z[3]);
      }
#pragma unroll
      for (int c = 0; c < C; ++c) st.v[tt][(p & 15) * C + c] = Cvt<T>::to_f32(fl.v[slot][tt][(p & 15) * C + c]);
      if constexpr (RULE == kDelta) {
        if ((p & 15) == 0) st.beta[tt] = logistic(Cvt<T>::to_f32(rb));
      }
    };
#pragma unroll
    for (int s = 0; s < kDepth; ++s) fetch(s);
    scalars(0);
    commit(0);
    fetch(kDepth);
    scalars(1);
    __syncthreads();
    for (int s = 0; s < n_stages; ++s) {
      commit(s + 1);                 // the other buffer: its readers passed the last barrier
      fetch(s + 1 + kDepth);
      scalars(s + 2);
      __syncthreads();
    }
    return;
  }

  // ---- the warps that own columns -------------------------------------------------------------------------------------------
  constexpr int NJ = DK / 32;          // groups of four rows per lane
  const int lane = threadIdx.x & 31, r = lane & 7, cg = lane >> 3;
  const int cw = warp * 4 * C + cg * C;               // first of the lane's columns within the CTA
  const int col = col_cta + cw;
  float* sp = A.state + (static_cast<int64_t>(sq.slot) * H + h) * dk * dv;
  f32x2 S[C][2 * NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float x[4][C];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = 32 * j + 4 * r + i;
#pragma unroll
      for (int c = 0; c < C; ++c) x[i][c] = 0.f;
      if (!sq.fresh && row < dk) {
        const float* src = sp + static_cast<int64_t>(row) * dv + col;
        if (C == 4 && A.vec_s) {
          if (col < dv) {
            const float4 f = *reinterpret_cast<const float4*>(src);
            x[i][0] = f.x, x[i][1 % C] = f.y, x[i][2 % C] = f.z, x[i][3 % C] = f.w;
          }
        } else {
#pragma unroll
          for (int c = 0; c < C; ++c) {
            if (col + c < dv) x[i][c] = src[c];
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      S[c][2 * j] = pair(x[0][c], x[1][c]);
      S[c][2 * j + 1] = pair(x[2][c], x[3][c]);
    }
  }
  const f32x2 dd = RULE == kRetention ? pair(A.decay[h], A.decay[h]) : 0ull;
  constexpr int kTok = 8 / C;          // tokens whose read-outs are reduced together
  const int my_t = r / C, my_c = r - my_t * C;
  const bool my_col = col + my_c < dv;
  float* op = A.o + (static_cast<int64_t>(sq.tok0) * H + h) * dv + col + my_c;
  const int64_t o_tok = static_cast<int64_t>(H) * dv;

  // a token's rows as this lane needs them: read while the token before is computed
  constexpr int kSections = S_t::kSections;
  struct Rows {
    f32x2 x[kSections][2 * NJ];      // q | f or k | 1 - f or g - 1
    float v[C], beta;
  };
  auto read = [&](Rows& r4, const S_t& st, int tt) {
    const float* row = st.rows[tt] + 4 * r;
#pragma unroll
    for (int n = 0; n < kSections; ++n) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(row + n * DK + 32 * j);
        r4.x[n][2 * j] = w.x, r4.x[n][2 * j + 1] = w.y;
      }
    }
    if constexpr (C == 4) {
      const float4 f = *reinterpret_cast<const float4*>(&st.v[tt][cw]);
      r4.v[0] = f.x, r4.v[1] = f.y, r4.v[2] = f.z, r4.v[3] = f.w;
    } else if constexpr (C == 2) {
      const float2 f = *reinterpret_cast<const float2*>(&st.v[tt][cw]);
      r4.v[0] = f.x, r4.v[1] = f.y;
    } else {
      r4.v[0] = st.v[tt][cw];
    }
    if constexpr (RULE == kDelta) r4.beta = st.beta[tt];
  };
  // The passes over the tile are written one after the other, every step of a pass on another pair: what a warp alone on its scheduler
  // waits for is the latency of dependent multiply-adds.
  auto token = [&](const Rows& in, float (&out)[C]) {
    f32x2 o2[C];
#pragma unroll
    for (int c = 0; c < C; ++c) o2[c] = 0ull;
    if constexpr (RULE == kDelta) {
      f32x2 d2[C];
#pragma unroll
      for (int c = 0; c < C; ++c) d2[c] = 0ull;
#pragma unroll
      for (int i = 0; i < 2 * NJ; ++i) {
#pragma unroll
        for (int c = 0; c < C; ++c) S[c][i] = fma2(in.x[2][i], S[c][i], S[c][i]);
      }
#pragma unroll
      for (int i = 0; i < 2 * NJ; ++i) {
#pragma unroll
        for (int c = 0; c < C; ++c) d2[c] = fma2(S[c][i], in.x[1][i], d2[c]);
      }
      float u[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const float2 f = halves(d2[c]);
        u[c] = f.x + f.y;
      }
#pragma unroll
      for (int x = 1; x < 8; x <<= 1) {
#pragma unroll
        for (int c = 0; c < C; ++c) u[c] += __shfl_xor_sync(0xffffffffu, u[c], x);
      }
      f32x2 uu[C];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        u[c] = in.beta * (in.v[c] - u[c]);
        uu[c] = pair(u[c], u[c]);
      }
#pragma unroll
      for (int i = 0; i < 2 * NJ; ++i) {
#pragma unroll
        for (int c = 0; c < C; ++c) S[c][i] = fma2(in.x[1][i], uu[c], S[c][i]);
      }
    } else {
      f32x2 vv[C];
#pragma unroll
      for (int c = 0; c < C; ++c) vv[c] = pair(in.v[c], in.v[c]);
#pragma unroll
      for (int i = 0; i < 2 * NJ; ++i) {
        f32x2 w[C];
#pragma unroll
        for (int c = 0; c < C; ++c) w[c] = mul2(in.x[RULE == kGated ? 2 : 1][i], vv[c]);
#pragma unroll
        for (int c = 0; c < C; ++c) S[c][i] = fma2(RULE == kGated ? in.x[1][i] : dd, S[c][i], w[c]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * NJ; ++i) {
#pragma unroll
      for (int c = 0; c < C; ++c) o2[c] = fma2(S[c][i], in.x[0][i], o2[c]);
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float2 f = halves(o2[c]);
      out[c] = f.x + f.y;
    }
  };
  // eight partial read-outs (token i / C, column i % C) of every lane -> lane r holds the sum of number r
  auto read_outs = [&](float (&part)[8]) {
    float a[4], b[2];
    const bool up4 = r & 4, up2 = r & 2, up1 = r & 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float give = up4 ? part[i] : part[i + 4], keep = up4 ? part[i + 4] : part[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float give = up2 ? a[i] : a[i + 2], keep = up2 ? a[i + 2] : a[i];
      b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const float give = up1 ? b[0] : b[1], keep = up1 ? b[1] : b[0];
    return keep + __shfl_xor_sync(0xffffffffu, give, 1);
  };

  __syncthreads();
  for (int s = 0; s < n_stages; ++s) {
    const S_t& st = stage[s & 1];
    const int n = min(kStage, sq.count - s * kStage);
    if (n == kStage) {
      Rows rows[2];
      read(rows[0], st, 0);
#pragma unroll
      for (int t0 = 0; t0 < kStage; t0 += kTok) {
        float part[8];
#pragma unroll
        for (int t = 0; t < kTok; ++t) {
          float o[C];
          if (t0 + t + 1 < kStage) read(rows[(t0 + t + 1) & 1], st, t0 + t + 1);
          token(rows[(t0 + t) & 1], o);
#pragma unroll
          for (int c = 0; c < C; ++c) part[t * C + c] = o[c];
        }
        const float o = read_outs(part);
        if (my_col) op[(s * kStage + t0 + my_t) * o_tok] = o;
      }
    } else {
#pragma unroll 1
      for (int t = 0; t < n; ++t) {
        float o[C], part[8];
        Rows one;
        read(one, st, t);
        token(one, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i] = i < C ? o[i < C ? i : 0] : 0.f;
        const float sum = read_outs(part);
        if (my_t == 0 && my_col) op[(s * kStage + t) * o_tok] = sum;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    float x[4][C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float2 lo = halves(S[c][2 * j]), hi = halves(S[c][2 * j + 1]);
      x[0][c] = lo.x, x[1][c] = lo.y, x[2][c] = hi.x, x[3][c] = hi.y;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = 32 * j + 4 * r + i;
      if (row >= dk) continue;
      float* dst = sp + static_cast<int64_t>(row) * dv + col;
      if (C == 4 && A.vec_s) {
        if (col < dv) *reinterpret_cast<float4*>(dst) = make_float4(x[i][0], x[i][1 % C], x[i][2 % C], x[i][3 % C]);
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (col + c < dv) dst[c] = x[i][c];
        }
      }
    }
  }
}

// Columns per lane: two give a lone warp per scheduler a shorter token, four read shared memory half as often; which is ahead changes
// with how many CTAs of two an SM gets (B200, 64 x 128 states, ns per token, gated / delta / retention; two against four columns): one
// 134 / 193 / 102 against 157 / 245 / 137, two 175 / 257 / 141 against 158 / 245 / 136, three 241 / 366 / 190 against 246 / 374 / 213, four
// 349 / 490 / 270 against 246 / 374 / 213, seven 555 / 805 / 434 against 469 / 721 / 405 (eight columns: 439 / 770 / 399, and 273 / 425 / 257
// from the first CTA on).  Keys of 65 .. 128 take four from two CTAs on without a table of their own; sizes whose tile would not fit the
// registers take fewer.
template <int RULE, typename T, int DK>
int launch_columns(ColArgs& A, int n_seqs, cudaStream_t stream, const char* name) {
  auto go = [&](auto cols) {
    constexpr int C = decltype(cols)::value;
    const dim3 grid(n_seqs, A.H, (A.dv + 4 * C * kColWarps - 1) / (4 * C * kColWarps));
    constexpr size_t smem = column_smem<RULE, T, DK, C>();
    auto kern = column_scan_kernel<RULE, T, DK, C>;
    if constexpr (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    kern<<<grid, kColNT, smem, stream>>>(A);
    return check_launch(name);
  };
  const int64_t columns = static_cast<int64_t>(n_seqs) * A.H * A.dv;
  const int64_t per_sm = (columns + 32 * kNumSMs - 1) / (32 * kNumSMs);
  if constexpr (DK <= 64) {
    if (per_sm != 1 && per_sm != 3) return go(std::integral_constant<int, 4>{});
  } else if constexpr (DK <= 128) {
    if (per_sm > 1) return go(std::integral_constant<int, 4>{});
  }
  if constexpr (DK <= 256) {
    return go(std::integral_constant<int, 2>{});
  } else {
    return go(std::integral_constant<int, 1>{});
  }
}

template <typename T>
void set_vec(ColArgs& A) {
  auto four = [](const void* p, int64_t stride) {
    return reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T)) == 0 && stride % 4 == 0;
  };
  A.vec_qk = four(A.in.q, A.in.stride) && four(A.in.k, A.in.stride) && A.dk % 4 == 0;
  A.vec_a = A.a && four(A.a, A.a_stride) && A.dk % 4 == 0;
  A.vec_v = four(A.in.v, A.in.stride) && A.dv % 4 == 0;
  A.vec_s = aligned16(A.state) && A.dv % 4 == 0;
}

template <int RULE>
int launch_rule(ColArgs& A, int n_seqs, int dtype, cudaStream_t stream, const char* name) {
  auto sized = [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    set_vec<T>(A);
    if (A.dk <= 32) return launch_columns<RULE, T, 32>(A, n_seqs, stream, name);
    if (A.dk <= 64) return launch_columns<RULE, T, 64>(A, n_seqs, stream, name);
    if (A.dk <= 128) return launch_columns<RULE, T, 128>(A, n_seqs, stream, name);
    if (A.dk <= 256) return launch_columns<RULE, T, 256>(A, n_seqs, stream, name);
    if constexpr (RULE != kDelta) {
      if (A.dk <= 512) return launch_columns<RULE, T, 512>(A, n_seqs, stream, name);
    }
    return fail(B200_ESHAPE, "%s: key size %d too large", name, A.dk);
  };
  switch (dtype) {
    case B200_DTYPE_F16:
      return sized(static_cast<__half*>(nullptr));
    case B200_DTYPE_BF16:
      return sized(static_cast<__nv_bfloat16*>(nullptr));
    case B200_DTYPE_F32:
      return sized(static_cast<float*>(nullptr));
    default:
      return fail(B200_EINVAL, "%s: unsupported dtype %d", name, dtype);
  }
}

ColArgs common_args(float* o, const ScanRows& in, float* state, const int32_t* seqs, const ScanShape& n) {
  ColArgs A{};
  A.o = o;
  A.in = in;
  A.state = state;
  A.seqs = reinterpret_cast<const ColSeq*>(seqs);
  A.H = n.H, A.G = n.G, A.dk = n.dk, A.dv = n.dv;
  return A;
}

}  // namespace

int gated_column_scan(float* o, const ScanRows& in, const void* f_bias, const void* lower, float* state, const int32_t* seqs,
                      const ScanShape& n, int dtype, cudaStream_t stream) {
  ColArgs A = common_args(o, in, state, seqs, n);
  A.bias = f_bias;
  A.rate = lower;
  return launch_rule<kGated>(A, n.n_seqs, dtype, stream, "b200_gated_scan");
}

int delta_column_scan(float* o, const ScanRows& in, const void* beta, int64_t beta_stride, const void* a, int64_t a_stride,
                      const void* dt_bias, const void* a_log, bool per_channel, float* state, const int32_t* seqs,
                      const ScanShape& n, float unit_eps, float q_scale, int dtype, cudaStream_t stream) {
  ColArgs A = common_args(o, in, state, seqs, n);
  A.beta = beta, A.beta_stride = beta_stride;
  A.a = a, A.a_stride = a_stride;
  A.bias = dt_bias;
  A.rate = a_log;
  A.per_channel = per_channel;
  A.unit_eps = unit_eps, A.scale = q_scale;
  return launch_rule<kDelta>(A, n.n_seqs, dtype, stream, "b200_delta_scan");
}

int retention_column_scan(float* o, const ScanRows& in, const float* decay, float k_scale, float* state, const int32_t* seqs,
                          const ScanShape& n, int dtype, cudaStream_t stream) {
  ColArgs A = common_args(o, in, state, seqs, n);
  A.decay = decay;
  A.scale = k_scale;
  return launch_rule<kRetention>(A, n.n_seqs, dtype, stream, "b200_retention_scan");
}

}  // namespace b200
