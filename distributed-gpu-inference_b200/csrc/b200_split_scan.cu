// The gated, delta and retention recurrences of b200_column_scan.cu over prompt portions of 16-bit inputs in chunks of 16 tokens on the
// tensor cores, at fp32 precision.  With f_t the decays of a chunk's tokens per key channel, F_t = f_1 .. f_t, S the fp32 state at its
// start, and every product of decays one of consecutive tokens (never a quotient: nothing overflows however fast a head forgets),
//
//   o_t = S^T (F_t q_t) + sum_(s <= t) P_ts v_s          P_ts = sum_i q_ti (f_(s+1) .. f_t)_i k_si
//   S  <- F_16 S + sum_s (f_(s+1) .. f_16 k_s) v_s^T
//
// (gated: k = 1 - f).  The delta rule writes u_s in the place of v_s, U = M (V - (F K) S) with M = (1 + A)^-1 diag(beta), A_ts = beta_t
// k_t (f_(s+1) .. f_t) k_s for s < t: the inverse of a unit lower triangle does not depend on the state.
//
// split_prepare_kernel makes a chunk's operands for every (chunk, head) of a step at once - activations, decays and their products, pair
// weights, the inverse - and leaves them in a workspace in the order in which the lanes of a warp hold them as B fragments;
// split_chain_kernel then walks the chunks of a (sequence, head, 64 value columns) in order.  A warp of it owns 16 value columns: S^T as
// eight accumulator tiles, which are as they lie (split) the A fragments of S^T (F q)^T.
//
// Precision.  Every fp32 operand x enters the products as three bf16 numbers (hi + mid + lo = x to 2^-25: each takes 8 bits of what is
// left), bf16 values as themselves, fp16 values as two; of the nine products of two split operands the three below 2^-24 are left out.
// Products of decays carry what their roundings lost.  A tensor-core accumulator rounds towards zero, so the leading products of every
// 16 channels are added up in fp32, and so is the state.  Values beyond 2^48, infinities and NaN (and decays beyond 1) have no such split:
// a (sequence, head) that holds one walks token by token in fp32, so that such a value reaches what it reaches there.  Against 64 bits
// (relative 2-norm, bf16 inputs, portions of 1 .. 700 tokens; token by token / here): gated read-outs 6.50e-8 / 6.57e-8, state 9.3e-8 /
// 7.0e-8; delta 1.31e-7 / 1.29e-7, 8.2e-8 / 8.1e-8; retention 3.8e-7 / 1.2e-7, 4.2e-7 / 1.1e-7.
//
// What bounds it.  The chain: latency - a chunk takes a lone warp per scheduler 1550 clocks (gated) and 2450 (delta) for 78 and 168
// products of 8 clocks each, between which its conversions (two clocks each) stand; the CTAs of an SM overlap (three of the segments' kernel, at 8 x
// 2048 tokens of 16 heads, which run in one piece but for that measurement: 1250 clocks a chunk, products 47 % of the time, issue slots as
// much).  Two warps per 16 columns, bulk copies and packed fp32 arithmetic were each slower.  Where
// sequences and heads leave SMs idle the gated and the retention rule walk segments of a sequence at the same time (split_chain_kernel).  The
// operands: issue slots and accesses to shared memory, three quarters of both, at eight CTAs per SM.
// B200, bf16, 64 x 128 states, us token by token / here (operands + chain): gated, 6 portions of up to 1780 tokens of 16 heads 395 / 212
// (64 + 148), 1 of 2048 of 4 heads 132 / 36 (in one piece 124); delta, 8 x 2048 of 8 heads 467 / 290 (118 + 172; columns of P on eight lanes each, whose
// reads of a row four columns repeat, and the operands copied out by the threads: 138); retention, 5 x 1024 of 16 heads 184 / 98 (25 + 73).
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <type_traits>

#include "../../include/b200_mixers.h"
#include "b200_common.cuh"

namespace b200 {
namespace {

enum Rule { kGated, kDelta, kRetention };

struct SplitSeq {
  int tok0, count, slot, fresh;
};

constexpr int kTok = 16;         // tokens per chunk
constexpr int kDK = 64;          // key channels (smaller sizes are padded with zeros)
constexpr float kWild = 281474976710656.0f;   // 2^48

// One chunk's operands.  Fragments of B, [lane][register], three parts each: `q` (F q) and `fk` (F k, delta): channels 16 kk .. + 15 as
// the contraction, registers 0, 1 tokens 0 .. 7 and 2, 3 tokens 8 .. 15; `k` (keys times the decays behind them): tokens as the
// contraction, registers 0, 1 channels 16 kk .. + 7 and 2, 3 the next eight; `p`, `m`: P and M, source tokens as the contraction.
struct OpsBase {
  uint4 q[3][4][32];
  uint4 k[3][4][32];
  uint4 p[3][32];
  float f_end[2][kDK];       // F_16 as two floats
};
struct OpsDelta : OpsBase {
  uint4 fk[3][4][32];
  uint4 m[3][32];
};
template <int RULE>
using Ops = std::conditional_t<RULE == kDelta, OpsDelta, OpsBase>;

struct SplitArgs {
  float* o;
  const void* q;
  const void* k;          // gated: the forget gate's logits
  const void* v;
  int64_t stride;
  const void* beta; int64_t beta_stride;
  const void* a; int64_t a_stride;
  const void* bias;       // gated: f_bias, delta: dt_bias
  const void* rate;       // gated: lower, delta: a_log
  const float* decay;     // retention
  float* state;
  const SplitSeq* seqs;
  unsigned char* ops;     // [chunks of the step][heads of this launch]
  int* wild;              // the same order: the chunk holds a value that has no split
  int n_seqs, n_chunks;   // n_chunks: a bound of the step's
  int h0, heads;          // heads of this launch
  int seg;                // chunks per segment (0: sequences in one piece), and where segments leave their ends: [slot][heads][64-column block]
  float* ends;
  int H, G, dk, dv;
  int per_channel;        // delta: a decay logit and a bias per key channel (1) or one per head (0)
  int vec_qk, vec_a, vec_c;   // eight elements of q / k, a, the constants can be read at once
  int vec_v;              // and of v: 8, 4 or 1
  float unit_eps, scale;  // delta: q_scale; retention: k_scale
};

__device__ __forceinline__ float soft_plus(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

using f32x2 = unsigned long long;
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

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {   // c = a b
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ uint32_t two(float lo, float hi) {   // bf16 pair, lo in the lower half
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float low(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float high(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
// x, y -> three bf16 pairs whose sums they are
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = two(x, y);
  x -= low(hi), y -= high(hi);
  mid = two(x, y);
  lo = two(x - low(mid), y - high(mid));
}
// x + dx, y + dy (dx, dy: below the last bits of x and y)
__device__ __forceinline__ void split3(float x, float y, float dx, float dy, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = two(x, y);
  x -= low(hi), y -= high(hi);
  mid = two(x, y);
  lo = two(x - low(mid) + dx, y - high(mid) + dy);
}
// Where lane L's registers of a fragment lie among the 32: eight consecutive lanes still cover all banks, and so do most of the words that
// a preparing warp writes at once (as they come: 16 lanes to a bank).
__device__ __forceinline__ int slot_of(int L, int kk) { return L ^ ((L >> 3) & 3) ^ ((kk & 1) << 2); }
__device__ __forceinline__ bool tame(float x) { return fabsf(x) < kWild; }   // false for NaN
__device__ __forceinline__ int chunks_of(int count) { return (max(count, 0) + kTok - 1) / kTok; }

// Chunks of the sequences before `seq` (a warp's work).
__device__ __forceinline__ int chunks_before(const SplitSeq* seqs, int seq) {
  int n = 0;
  for (int i = threadIdx.x & 31; i < seq; i += 32) n += chunks_of(seqs[i].count);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}
// The sequence that piece x of the step belongs to and its place in it, a sequence having `pieces` of them (a warp's work); false: beyond the last.
template <typename Pieces>
__device__ __forceinline__ bool find_piece(const SplitSeq* seqs, int n_seqs, int x, int& seq, int& place, Pieces pieces) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < n_seqs; base += 32) {
    const int n = base + lane < n_seqs ? pieces(seqs[base + lane]) : 0;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const unsigned past = __ballot_sync(0xffffffffu, sum > x);
    if (past) {
      const int who = __ffs(past) - 1;
      seq = base + who;
      place = x - __shfl_sync(0xffffffffu, sum - n, who);
      return true;
    }
    x -= __shfl_sync(0xffffffffu, sum, 31);
  }
  return false;
}

// Segments that a sequence has beyond its first.
__device__ __forceinline__ int extra_segments(const SplitSeq& s, int seg) { return (max(chunks_of(s.count), 1) - 1) / seg; }
// The place that the first extra segment of `seq` has among all (a warp's work).
__device__ __forceinline__ int extra_before(const SplitSeq* seqs, int seq, int seg) {
  int n = 0;
  for (int i = threadIdx.x & 31; i < seq; i += 32) n += extra_segments(seqs[i], seg);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  return n;
}

// Eight elements of a row from channel e on, `left` of which exist.
template <typename T>
__device__ __forceinline__ void read8(float (&d)[8], const T* p, int left, bool vec) {
  alignas(16) T e[8];
  if (vec && left >= 8) {
    *reinterpret_cast<uint4*>(e) = *reinterpret_cast<const uint4*>(p);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = i < left ? p[i] : Cvt<T>::from_f32(0.f);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) d[i] = Cvt<T>::to_f32(e[i]);
}

// A token's q, k and decays (delta: decays - 1) of eight channels from the raw rows; `sum8` adds over a token's threads.
template <int RULE, typename T, typename Sum>
__device__ __forceinline__ void activate(const SplitArgs& A, int h, int e0, float ret, float (&x)[8], float (&y)[8], float (&z)[8], Sum sum8) {
  if constexpr (RULE == kDelta) {
    float sq = 0.f, sk = 0.f, b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) sq = fmaf(x[i], x[i], sq), sk = fmaf(y[i], y[i], sk);
    sq = rsqrtf(sum8(sq) + A.unit_eps) * A.scale;
    sk = rsqrtf(sum8(sk) + A.unit_eps);
    const float a_rate = expf(Cvt<T>::to_f32(static_cast<const T*>(A.rate)[h]));
    if (A.per_channel) {
      read8(b, static_cast<const T*>(A.bias) + h * A.dk + e0, A.dk - e0, A.vec_c);
    } else {
      const float one = Cvt<T>::to_f32(static_cast<const T*>(A.bias)[h]);
#pragma unroll
      for (int i = 0; i < 8; ++i) b[i] = one;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[i] *= sq, y[i] *= sk;
      z[i] = e0 + i < A.dk ? expm1f(-a_rate * soft_plus(z[i] + b[i])) : 0.f;
    }
  } else if constexpr (RULE == kGated) {
    float b[8], l[8];
    read8(b, static_cast<const T*>(A.bias) + h * A.dk + e0, A.dk - e0, A.vec_c);
    read8(l, static_cast<const T*>(A.rate) + h * A.dk + e0, A.dk - e0, A.vec_c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // f and 1 - f each to their own last digits: 1 minus a rounded f near 1 would lose most of them, and f as 1 minus a k near 1
      const float u = y[i] + b[i], k = (1.0f - l[i]) * row_logistic(-u), f = l[i] + (1.0f - l[i]) * row_logistic(u);
      x[i] *= row_logistic(x[i]);
      y[i] = e0 + i < A.dk ? k : 0.f;
      z[i] = e0 + i < A.dk ? (f < 0.5f ? f : 1.0f - k) : 0.f;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] *= A.scale, z[i] = ret;
  }
}

// ---- operands -----------------------------------------------------------------------------------------------------------------------
template <int RULE>
struct Prep {
  Ops<RULE> ops;
  alignas(16) float rows[RULE == kRetention ? 2 : 3][kTok][kDK];   // q | k | decays (delta: minus one)
  alignas(16) float p[kTok][kTok + 4];
  alignas(16) float a[RULE == kDelta ? kTok : 1][kTok + 4];
  float beta[kTok];
};

template <int RULE, typename T>
__global__ void __launch_bounds__(128)
split_prepare_kernel(const SplitArgs A) {
  extern __shared__ __align__(16) unsigned char prep_raw[];
  Prep<RULE>& sm = *reinterpret_cast<Prep<RULE>*>(prep_raw);
  int seq, place;
  if (!find_piece(A.seqs, A.n_seqs, blockIdx.x, seq, place, [](const SplitSeq& s) { return chunks_of(s.count); })) return;
  const SplitSeq sq = A.seqs[seq];
  const int h = A.h0 + blockIdx.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_live = min(kTok, sq.count - place * kTok);
  const float ret = RULE == kRetention ? A.decay[h] : 0.f;

  // rows: eight threads per token, eight channels each.  Dead tokens: q = k = 0, decays of 1.
  float big = 0.f, most = 0.f;     // squares of everything that is split, the largest decay
  {
    const int tt = threadIdx.x >> 3, e0 = (threadIdx.x & 7) * 8;
    const bool live = tt < n_live;
    const int64_t tok = sq.tok0 + place * kTok + min(tt, n_live - 1);
    const int gq = h / (A.H / A.G);
    float x[8], y[8], z[8];
    read8(x, static_cast<const T*>(A.q) + tok * A.stride + gq * A.dk + e0, A.dk - e0, A.vec_qk);
    read8(y, static_cast<const T*>(A.k) + tok * A.stride + gq * A.dk + e0, A.dk - e0, A.vec_qk);
    float raw_beta = 0.f;
    if constexpr (RULE == kDelta) {
      if (A.per_channel) {
        read8(z, static_cast<const T*>(A.a) + tok * A.a_stride + h * A.dk + e0, A.dk - e0, A.vec_a);
      } else {
        const float one = Cvt<T>::to_f32(static_cast<const T*>(A.a)[tok * A.a_stride + h]);
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = one;
      }
      raw_beta = Cvt<T>::to_f32(static_cast<const T*>(A.beta)[tok * A.beta_stride + h]);
    }
    for (int c0 = e0; c0 < A.dv; c0 += kDK) {
      float f[8];
      read8(f, static_cast<const T*>(A.v) + tok * A.stride + static_cast<int64_t>(h) * A.dv + c0, A.dv - c0, A.vec_v == 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) big = fmaf(f[i], f[i], big);
    }
    activate<RULE, T>(A, h, e0, ret, x, y, z, [](float s) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      return s;
    });
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      big = fmaf(x[i], x[i], fmaf(y[i], y[i], fmaf(z[i], z[i], big)));
      most = fmaxf(most, fabsf(z[i]));
      if (!live) x[i] = y[i] = 0.f, z[i] = RULE == kDelta ? 0.f : 1.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      *reinterpret_cast<float4*>(&sm.rows[0][tt][e0 + i]) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
      *reinterpret_cast<float4*>(&sm.rows[1][tt][e0 + i]) = make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]);
      if constexpr (RULE != kRetention) *reinterpret_cast<float4*>(&sm.rows[2][tt][e0 + i]) = make_float4(z[i], z[i + 1], z[i + 2], z[i + 3]);
    }
    if constexpr (RULE == kDelta) {
      const float b = row_logistic(raw_beta);
      big = fmaf(b, b, big);
      if (e0 == 0) sm.beta[tt] = live ? b : 0.f;
    }
  }
  const bool ok = big < kWild * kWild && most < 1.001f;      // false for NaN
  const int any = __syncthreads_or(!ok);

  // Columns of P (and of A), four to a warp: sixteen lanes share two, four channels each, so that a row of the tokens is read once for both; the
  // decayed keys walk down the tokens
  {
    const int s0 = 4 * w + 2 * (lane >> 4), c = lane & 15;
    auto load4 = [&](f32x2 (&d)[2], const float* row) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(row + 4 * c);
      d[0] = x.x, d[1] = x.y;
    };
    auto dot4 = [](const f32x2 (&x)[2], const f32x2 (&y)[2]) {
      const float2 a = halves(fma2(x[1], y[1], mul2(x[0], y[0])));
      return a.x + a.y;
    };
    // eight partial sums of every lane -> lanes 2 i and 2 i + 1 of the sixteen hold the sum of number i
    auto sums = [&](const float (&v)[8]) {
      const bool up8 = c & 8, up4 = c & 4, up2 = c & 2;
      float a[4], b[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float give = up8 ? v[i] : v[i + 4], keep = up8 ? v[i + 4] : v[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float give = up4 ? a[i] : a[i + 2], keep = up4 ? a[i + 2] : a[i];
        b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
      }
      const float give = up2 ? b[0] : b[1], keep = up2 ? b[1] : b[0];
      const float d = keep + __shfl_xor_sync(0xffffffffu, give, 2);
      return d + __shfl_xor_sync(0xffffffffu, d, 1);
    };
    f32x2 kw[2][2];
    load4(kw[0], sm.rows[1][s0]);
    load4(kw[1], sm.rows[1][s0 + 1]);
    auto block = [&](int t0, auto own) {          // four tokens; `own`: the block of the columns themselves
      constexpr bool kOwn = decltype(own)::value;
      float part[8];
      [[maybe_unused]] float part_a[RULE == kDelta ? 8 : 1];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = t0 + i;
        f32x2 x[2];
        if (!kOwn || i > 0) {
          if constexpr (RULE != kRetention) load4(x, sm.rows[RULE == kRetention ? 0 : 2][t]);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const bool decays = !kOwn || t > s0 + u;
            [[maybe_unused]] const uint32_t f = __float_as_uint(decays && t < n_live ? ret : 1.0f);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              if constexpr (RULE == kRetention) kw[u][j] = mul2(kw[u][j], static_cast<f32x2>(f) << 32 | f);
              else if constexpr (RULE == kDelta) kw[u][j] = fma2(kw[u][j], decays ? x[j] : 0ull, kw[u][j]);
              else kw[u][j] = mul2(kw[u][j], decays ? x[j] : 0x3f8000003f800000ull);
            }
          }
        }
        load4(x, sm.rows[0][t]);
#pragma unroll
        for (int u = 0; u < 2; ++u) part[4 * u + i] = !kOwn || t >= s0 + u ? dot4(kw[u], x) : 0.f;
        if constexpr (RULE == kDelta) {
          load4(x, sm.rows[1][t]);
#pragma unroll
          for (int u = 0; u < 2; ++u) part_a[4 * u + i] = !kOwn || t > s0 + u ? dot4(kw[u], x) : 0.f;
        }
      }
      const int t = t0 + ((c >> 1) & 3), s = s0 + (c >> 3);
      const float p = sums(part);
      if ((c & 1) == 0) sm.p[t][s] = p;
      if constexpr (RULE == kDelta) {
        const float a = sums(part_a);
        if ((c & 1) == 0) sm.a[t][s] = sm.beta[t] * a;
      }
    };
    for (int t = c >> 1; t < 4 * w; t += 8) {
      const int s = s0 + (c & 1);
      sm.p[t][s] = 0.f;
      if constexpr (RULE == kDelta) sm.a[t][s] = 0.f;
    }
    block(4 * w, std::true_type{});
#pragma unroll 1
    for (int t0 = 4 * w + 4; t0 < kTok; t0 += 4) block(t0, std::false_type{});
  }
  // Products of decays as two floats each, channels 2 lane and 2 lane + 1.
  const int e = 2 * lane;
  float2 F = make_float2(1.f, 1.f), F_lo = make_float2(0.f, 0.f);
  auto at = [&](int section, int t) { return *reinterpret_cast<const float2*>(&sm.rows[section][t][e]); };
  auto times1 = [](float& hi, float& lo, float z, float k) {
    float f = z, lost = 0.f;
    if constexpr (RULE == kDelta) {            // 1 + (g - 1), and what the sum lost
      f = 1.0f + z;
      lost = z - (f - 1.0f);
    } else if constexpr (RULE == kGated) {     // f from 1/2 on is a rounded 1 - k: what the difference lost
      lost = f < 0.5f ? 0.f : (1.0f - f) - k;
    }
    const float p = hi * f;
    lo = fmaf(lo, f, fmaf(hi, f, RULE == kRetention ? -p : fmaf(hi, lost, -p)));
    hi = p;
  };
  auto times = [&](int t) {
    const float f = t < n_live ? ret : 1.0f;
    const float2 z = RULE == kRetention ? make_float2(f, f) : at(RULE == kRetention ? 0 : 2, t), k = RULE == kGated ? at(1, t) : z;
    times1(F.x, F_lo.x, z.x, k.x);
    times1(F.y, F_lo.y, z.y, k.y);
  };
  auto scaled = [&](float2 x, float2& p, float2& d) {       // x F and what its rounding lost
    p = make_float2(x.x * F.x, x.y * F.y);
    d = make_float2(fmaf(x.x, F_lo.x, fmaf(x.x, F.x, -p.x)), fmaf(x.y, F_lo.y, fmaf(x.y, F.y, -p.y)));
  };
  auto put = [](uint4* part0, int part, int lane_of, int reg, float x, float y, float dx, float dy) {
    uint32_t hi, mid, lo;
    split3(x, y, dx, dy, hi, mid, lo);
    uint32_t* to = reinterpret_cast<uint32_t*>(part0 + lane_of) + reg;
    to[0] = hi, to[4 * part] = mid, to[8 * part] = lo;
  };
  if (w == 0 || w == 2) {            // F q (and F k): tokens 8 half .. + 7
    const int half = w >> 1;
    for (int t = 0; t < 8 * half; ++t) times(t);
#pragma unroll 4
    for (int i = 0; i < 8; ++i) {
      const int t = 8 * half + i;
      times(t);
      const int to = slot_of(4 * i + (lane & 3), lane >> 3), reg = ((lane >> 2) & 1) + 2 * half;
      float2 p, d;
      scaled(at(0, t), p, d);
      put(sm.ops.q[0][lane >> 3], 128, to, reg, p.x, p.y, d.x, d.y);
      if constexpr (RULE == kDelta) {
        scaled(at(1, t), p, d);
        put(sm.ops.fk[0][lane >> 3], 128, to, reg, p.x, p.y, d.x, d.y);
      }
    }
    if (half == 1) {
      *reinterpret_cast<float2*>(&sm.ops.f_end[0][e]) = F;
      *reinterpret_cast<float2*>(&sm.ops.f_end[1][e]) = F_lo;
    }
  } else {                           // keys times the decays behind them: tokens 8 half .. + 7, from the last to the first
    const int half = w == 1;
    for (int t = kTok - 1; t > 8 * half + 7; --t) times(t);
#pragma unroll 2
    for (int i = 6; i >= 0; i -= 2) {
      const int t = 8 * half + i;
      float2 p1, d1, p0, d0;
      scaled(at(1, t + 1), p1, d1);
      times(t + 1);
      scaled(at(1, t), p0, d0);
      times(t);
      // channel 2 lane: tile (lane / 4), row (2 lane) % 8
      const int reg = half + 2 * ((lane >> 2) & 1), row = e & 7;
      put(sm.ops.k[0][lane >> 3], 128, slot_of(4 * row + (i >> 1), lane >> 3), reg, p0.x, p1.x, d0.x, d1.x);
      put(sm.ops.k[0][lane >> 3], 128, slot_of(4 * (row + 1) + (i >> 1), lane >> 3), reg, p0.y, p1.y, d0.y, d1.y);
    }
  }
  __syncthreads();
  if constexpr (RULE == kDelta) {
    // M = (1 + A)^-1 diag(beta): lane s < 16 of the first warp owns column s, in the place of A
    if (w == 0) {
      const int s = lane & 15;
      const float b = sm.beta[s];
      float x[kTok];
#pragma unroll
      for (int t = 0; t < kTok; ++t) {
        float a[4] = {t == s ? 1.0f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < t; r += 4) {
          const float4 l = *reinterpret_cast<const float4*>(&sm.a[t][r]);
          a[0] = fmaf(-l.x, x[r], a[0]);
          if (r + 1 < t) a[1] = fmaf(-l.y, x[r + 1], a[1]);
          if (r + 2 < t) a[2] = fmaf(-l.z, x[r + 2], a[2]);
          if (r + 3 < t) a[3] = fmaf(-l.w, x[r + 3], a[3]);
        }
        x[t] = (a[0] + a[1]) + (a[2] + a[3]);
      }
      __syncwarp();
      if (lane < kTok) {
#pragma unroll
        for (int t = 0; t < kTok; ++t) sm.a[t][s] = x[t] * b;
      }
    }
    __syncthreads();
  }
  {
    const int t = threadIdx.x >> 3, s = 2 * (threadIdx.x & 7);
    const int to = slot_of(4 * (t & 7) + ((s & 7) >> 1), 0), reg = (s >> 3) + 2 * (t >> 3);
    put(sm.ops.p[0], 32, to, reg, sm.p[t][s], sm.p[t][s + 1], 0.f, 0.f);
    if constexpr (RULE == kDelta) put(sm.ops.m[0], 32, to, reg, sm.a[t][s], sm.a[t][s + 1], 0.f, 0.f);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) {      // out by the copy engine
    const int64_t place_of = static_cast<int64_t>(blockIdx.x) * A.heads + blockIdx.y;
    static_assert(sizeof(Ops<RULE>) % 16 == 0 && alignof(Ops<RULE>) % 16 == 0);      // what the copy asks of both ends
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(A.ops + place_of * static_cast<int64_t>(sizeof(Ops<RULE>))), "r"(smem_addr(&sm.ops)),
                 "n"(sizeof(Ops<RULE>)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    A.wild[place_of] = any;
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
}

// ---- token by token, for a (sequence, head) that holds a value without a split: a warp owns 16 columns, lane (r, c)
// channels 8 j + 2 c, + 1 of its two ------------------------------------------------------------------------------------------------
template <int RULE, typename T>
__device__ __forceinline__ void walk_tokens(const SplitArgs& A, const SplitSeq& sq, int h, float* sp, float* op, const T* vp, int v_col, bool in0,
                                         bool in1, float* rows) {   // sp, op: at the first of the columns; v_col: its place in vp
  const int c = threadIdx.x & 3, dk = A.dk, dv = A.dv, gq = h / (A.H / A.G);
  const float ret = RULE == kRetention ? A.decay[h] : 0.f;
  const int64_t o_tok = static_cast<int64_t>(A.H) * dv;
  float S[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = 8 * j + 2 * c + (i & 1);
      S[j][i] = !sq.fresh && e < dk && (i >> 1 ? in1 : in0) ? sp[static_cast<int64_t>(e) * dv + 8 * (i >> 1)] : 0.f;
    }
  }
  auto quad = [](float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
  };
#pragma unroll 1
  for (int t = 0; t < sq.count; ++t) {
    const int64_t tok = sq.tok0 + t;
    float* row = rows + (t & 1) * 4 * kDK;     // q | k | decays | beta, made by the first eight threads
    if (threadIdx.x < 8) {
      const int e0 = 8 * threadIdx.x;
      float x[8], y[8], z[8];
      read8(x, static_cast<const T*>(A.q) + tok * A.stride + gq * dk + e0, dk - e0, false);
      read8(y, static_cast<const T*>(A.k) + tok * A.stride + gq * dk + e0, dk - e0, false);
      if constexpr (RULE == kDelta) {
        if (A.per_channel) {
          read8(z, static_cast<const T*>(A.a) + tok * A.a_stride + h * dk + e0, dk - e0, false);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) z[i] = Cvt<T>::to_f32(static_cast<const T*>(A.a)[tok * A.a_stride + h]);
        }
        if (e0 == 0) row[3 * kDK] = row_logistic(Cvt<T>::to_f32(static_cast<const T*>(A.beta)[tok * A.beta_stride + h]));
      }
      activate<RULE, T>(A, h, e0, ret, x, y, z, [](float s) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffu, s, o);
        return s;
      });
#pragma unroll
      for (int i = 0; i < 8; ++i) row[e0 + i] = x[i], row[kDK + e0 + i] = y[i], row[2 * kDK + e0 + i] = z[i];
    }
    __syncthreads();
    float v0 = in0 ? Cvt<T>::to_f32(vp[t * A.stride + v_col]) : 0.f, v1 = in1 ? Cvt<T>::to_f32(vp[t * A.stride + v_col + 8]) : 0.f;
    auto at = [&](int section, int j) { return *reinterpret_cast<const float2*>(row + section * kDK + 8 * j + 2 * c); };
    if constexpr (RULE == kDelta) {
      float u0 = 0.f, u1 = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 g = at(2, j), k = at(1, j);
        S[j][0] = fmaf(g.x, S[j][0], S[j][0]), S[j][1] = fmaf(g.y, S[j][1], S[j][1]);
        S[j][2] = fmaf(g.x, S[j][2], S[j][2]), S[j][3] = fmaf(g.y, S[j][3], S[j][3]);
        u0 = fmaf(S[j][0], k.x, fmaf(S[j][1], k.y, u0)), u1 = fmaf(S[j][2], k.x, fmaf(S[j][3], k.y, u1));
      }
      v0 = row[3 * kDK] * (v0 - quad(u0)), v1 = row[3 * kDK] * (v1 - quad(u1));
    }
    float o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 k = at(1, j), q = at(0, j);
      const float2 f = RULE == kDelta ? make_float2(1.0f, 1.0f) : at(2, j);
      S[j][0] = fmaf(f.x, S[j][0], k.x * v0), S[j][1] = fmaf(f.y, S[j][1], k.y * v0);
      S[j][2] = fmaf(f.x, S[j][2], k.x * v1), S[j][3] = fmaf(f.y, S[j][3], k.y * v1);
      o0 = fmaf(S[j][0], q.x, fmaf(S[j][1], q.y, o0)), o1 = fmaf(S[j][2], q.x, fmaf(S[j][3], q.y, o1));
    }
    o0 = quad(o0), o1 = quad(o1);
    if (c == 0 && in0) op[t * o_tok] = o0;
    if (c == 1 && in1) op[t * o_tok + 8] = o1;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = 8 * j + 2 * c + (i & 1);
      if (e < dk && (i >> 1 ? in1 : in0)) sp[static_cast<int64_t>(e) * dv + 8 * (i >> 1)] = S[j][i];
    }
  }
}

// ---- the chain ----------------------------------------------------------------------------------------------------------------------
constexpr int kStages = 3;
constexpr int kCols = 64;              // value columns of a CTA
constexpr int kChainNT = 2 * kCols;
constexpr int kEnd = kChainNT * 32 + 2 * kDK;     // floats of a segment's end: the state as its threads hold it, the product of its decays as two floats
template <int RULE, typename T>
struct Stage {
  Ops<RULE> ops;
  alignas(16) T v[kTok][kCols + 8];
};
template <int RULE, typename T>
struct Chain {
  Stage<RULE, T> stages[kStages];
};

using Tiles = float[2][4];           // accumulator tiles, of eight tokens or channels each
struct Split {
  uint32_t hi[4], mid[4], lo[4];
};
struct B3 {
  uint4 hi, mid, lo;
};
__device__ __forceinline__ void split_tiles(Split& s, const float (&x)[4], const float (&y)[4]) {      // two accumulator tiles -> an A fragment
  split3(x[0], x[1], s.hi[0], s.mid[0], s.lo[0]);
  split3(x[2], x[3], s.hi[1], s.mid[1], s.lo[1]);
  split3(y[0], y[1], s.hi[2], s.mid[2], s.lo[2]);
  split3(y[2], y[3], s.hi[3], s.mid[3], s.lo[3]);
}
__device__ __forceinline__ void add(Tiles& o, const Tiles& p) {
#pragma unroll
  for (int t = 0; t < 2; ++t) {
#pragma unroll
    for (int i = 0; i < 4; ++i) o[t][i] += p[t][i];
  }
}

// Two operands' six products with two tiles each.  The leading ones go to x, y, the small ones to s, t.  An accumulator's next product is
// four instructions on: what a product takes is covered by the three others.
__device__ __forceinline__ void mma6x2(Tiles& x, Tiles& y, Tiles& s, Tiles& t, const Split& a, const B3& b, const Split& c, const B3& d) {
  auto four = [](Tiles& x, Tiles& y, const uint32_t (&a)[4], const uint4& b, const uint32_t (&c)[4], const uint4& d) {
    mma(x[0], a, b.x, b.y), mma(x[1], a, b.z, b.w), mma(y[0], c, d.x, d.y), mma(y[1], c, d.z, d.w);
  };
  auto four_new = [](Tiles& x, Tiles& y, const uint32_t (&a)[4], const uint4& b, const uint32_t (&c)[4], const uint4& d) {
    mma_new(x[0], a, b.x, b.y), mma_new(x[1], a, b.z, b.w), mma_new(y[0], c, d.x, d.y), mma_new(y[1], c, d.z, d.w);
  };
  four_new(s, t, a.hi, b.lo, c.hi, d.lo);
  four(s, t, a.lo, b.hi, c.lo, d.hi);
  four(s, t, a.mid, b.mid, c.mid, d.mid);
  four(s, t, a.mid, b.hi, c.mid, d.hi);
  four(s, t, a.hi, b.mid, c.hi, d.mid);
  four_new(x, y, a.hi, b.hi, c.hi, d.hi);
}

// one operand's: the small ones in two chains
__device__ __forceinline__ void mma6(Tiles& x, Tiles& s, Tiles& t, const Split& a, const B3& b) {
  mma_new(s[0], a.hi, b.lo.x, b.lo.y), mma_new(s[1], a.hi, b.lo.z, b.lo.w);
  mma_new(t[0], a.lo, b.hi.x, b.hi.y), mma_new(t[1], a.lo, b.hi.z, b.hi.w);
  mma(s[0], a.mid, b.mid.x, b.mid.y), mma(s[1], a.mid, b.mid.z, b.mid.w);
  mma(t[0], a.mid, b.hi.x, b.hi.y), mma(t[1], a.mid, b.hi.z, b.hi.w);
  mma(s[0], a.hi, b.mid.x, b.mid.y), mma(s[1], a.hi, b.mid.z, b.mid.w);
  mma_new(x[0], a.hi, b.hi.x, b.hi.y), mma_new(x[1], a.hi, b.hi.z, b.hi.w);
}

// Four warps of 16 value columns each.
//
// Sequences in segments (A.seg; not the delta rule, whose decay is no diagonal): the first launch walks every sequence's first segment and, from a
// zero state and without read-outs, those between the first and the last; the second launch (`later`) starts the others from
// S <- F S + end over the segments before, F being a segment's product of decays.  The state pool is read by the first launch and
// written by the one that walks a sequence's last segment.
template <int RULE, typename T, int CTAS>
__global__ void __launch_bounds__(kChainNT, CTAS)
split_chain_kernel(const SplitArgs A, const bool later) {
  constexpr bool kHalfIn = std::is_same_v<T, __half>;
  using S_t = Stage<RULE, T>;
  extern __shared__ __align__(128) unsigned char chain_raw[];
  Chain<RULE, T>& sm = *reinterpret_cast<Chain<RULE, T>*>(chain_raw);
  int seq = blockIdx.x, seg = 0;
  const bool cut = RULE != kDelta && A.seg > 0;
  if (cut && (later || seq >= A.n_seqs)) {
    const int x = later ? seq : seq - A.n_seqs, per = A.seg;
    if (!find_piece(A.seqs, A.n_seqs, x, seq, seg, [per](const SplitSeq& s) { return extra_segments(s, per); })) return;
    ++seg;
  }
  const SplitSeq sq = A.seqs[seq];
  const int h = A.h0 + blockIdx.y, H = A.H, dk = A.dk, dv = A.dv;
  const int col_cta = blockIdx.z * kCols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_all = chunks_of(sq.count), last_seg = cut ? extra_segments(sq, A.seg) : 0;
  const int c0 = cut ? seg * A.seg : 0, n_chunks = cut ? min(A.seg, n_all - c0) : n_all;
  const int before = chunks_before(A.seqs, seq);
  const bool made = before + n_all <= A.n_chunks;      // sequences that share tokens may have more chunks than the workspace: no operands
  const int64_t first = static_cast<int64_t>(before + c0) * A.heads + blockIdx.y;
  // a segment's end: threads' states in float4s, then the decays.  The first segment of a cut sequence has 1 / 0 in their place: walked by tokens / not
  const int slot0_seg = last_seg > 0 ? extra_before(A.seqs, seq, A.seg) : 0;
  auto end_of = [&](int s) { return A.ends + ((static_cast<int64_t>(slot0_seg + s) * A.heads + blockIdx.y) * gridDim.z + blockIdx.z) * kEnd; };
  if (seg > 0 && (!made || (!later && seg == last_seg))) return;

  const int r = lane >> 2, c = lane & 3, m = lane >> 3, l8 = lane & 7;
  const int col = col_cta + 16 * warp + r;           // and col + 8
  const bool in0 = col < dv, in1 = col + 8 < dv;
  float* sp = A.state + (static_cast<int64_t>(sq.slot) * H + h) * dk * dv + col;
  float* op = A.o + (static_cast<int64_t>(sq.tok0) * H + h) * dv + col;
  const int64_t o_tok = static_cast<int64_t>(H) * dv;
  const T* vp = static_cast<const T*>(A.v) + sq.tok0 * A.stride + static_cast<int64_t>(h) * dv + col_cta;

  float S[8][4];          // S^T: columns col, col + 8; channels 8 j + 2 c, + 1
  auto leave_end = [&](float* end) {
#pragma unroll
    for (int j = 0; j < 8; ++j) reinterpret_cast<float4*>(end)[j * kChainNT + threadIdx.x] = make_float4(S[j][0], S[j][1], S[j][2], S[j][3]);
  };
  if (seg == 0) {
    bool odd = !made;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = 8 * j + 2 * c + (i & 1);
        S[j][i] = !sq.fresh && e < dk && (i >> 1 ? in1 : in0) ? sp[static_cast<int64_t>(e) * dv + 8 * (i >> 1)] : 0.f;
        odd = odd || !tame(S[j][i]);
      }
    }
    for (int i = threadIdx.x; made && i < n_all; i += kChainNT) odd = odd || A.wild[first + static_cast<int64_t>(i) * A.heads];
    odd = __syncthreads_or(odd);
    if (made && last_seg > 0 && threadIdx.x == 0) end_of(0)[kChainNT * 32] = odd ? 1.f : 0.f;
    if (odd) {
      walk_tokens<RULE, T>(A, sq, h, sp, op, vp, 16 * warp + r, in0, in1, reinterpret_cast<float*>(chain_raw));
      return;
    }
  } else if (later) {
    const float* end = end_of(0);
    if (end[kChainNT * 32] != 0.f) return;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 x = reinterpret_cast<const float4*>(end)[j * kChainNT + threadIdx.x];
      S[j][0] = x.x, S[j][1] = x.y, S[j][2] = x.z, S[j][3] = x.w;
    }
#pragma unroll 1
    for (int s = 1; s < seg; ++s) {
      end = end_of(s);
      const float* f = end + kChainNT * 32;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 x = reinterpret_cast<const float4*>(end)[j * kChainNT + threadIdx.x];
        const float2 hi = *reinterpret_cast<const float2*>(f + 8 * j + 2 * c), lo = *reinterpret_cast<const float2*>(f + kDK + 8 * j + 2 * c);
        S[j][0] = fmaf(S[j][0], hi.x, fmaf(S[j][0], lo.x, x.x)), S[j][1] = fmaf(S[j][1], hi.y, fmaf(S[j][1], lo.y, x.y));
        S[j][2] = fmaf(S[j][2], hi.x, fmaf(S[j][2], lo.x, x.z)), S[j][3] = fmaf(S[j][3], hi.y, fmaf(S[j][3], lo.y, x.w));
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) S[j][0] = S[j][1] = S[j][2] = S[j][3] = 0.f;
  }
  if (seg > 0) {
    op += static_cast<int64_t>(c0) * kTok * o_tok;
    vp += static_cast<int64_t>(c0) * kTok * A.stride;
  }
  const int n_tok = sq.count - c0 * kTok;      // from the segment's first on

  // what a thread copies of every chunk: 16-byte pieces of the operands, eight values of one token
  constexpr int kPieces = sizeof(Ops<RULE>) / 16;
  const uint4* src = reinterpret_cast<const uint4*>(A.ops + first * static_cast<int64_t>(sizeof(Ops<RULE>))) + threadIdx.x;
  const int64_t src_step = static_cast<int64_t>(A.heads) * kPieces;
  const int v_tok = threadIdx.x >> 3, v_col = 8 * (threadIdx.x & 7), v_left = dv - col_cta - v_col;
  const bool v_wide = A.vec_v == 8 && dv - col_cta >= kCols;      // the same for all
  const T* v_src = vp + static_cast<int64_t>(v_tok) * A.stride + v_col;
  auto fetch = [&](int q, int at, auto part) {        // called for q = 0, 1, 2 ..; `part`: what a state alone needs (k, and p behind it, to f_end)
    if (q < n_chunks) {
      constexpr int kFrom = decltype(part)::value ? offsetof(OpsBase, k) / 16 : 0;
      S_t& st = sm.stages[at];
      const uint32_t dst = smem_addr(&st.ops) + 16 * threadIdx.x;
#pragma unroll
      for (int i = kFrom; i < kPieces; i += kChainNT) {
        if (i + kChainNT <= kPieces || threadIdx.x < kPieces - i) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + i) : "memory");
      }
      src += src_step;
      const bool live = q * kTok + v_tok < n_tok;                 // zeros beyond the last token
      const T* from = live ? v_src : vp;
      T* to = &st.v[v_tok][v_col];
      if (v_wide) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(to)), "l"(from), "r"(live ? 16 : 0) : "memory");
      } else if (A.vec_v >= 4 && v_left >= 8) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(to)), "l"(from), "r"(live ? 8 : 0) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(to + 4)), "l"(from + 4), "r"(live ? 8 : 0) : "memory");
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) to[i] = live && i < v_left ? from[i] : Cvt<T>::from_f32(0.f);
      }
      v_src += kTok * A.stride;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int slot0 = slot_of(lane, 0), slot1 = slot_of(lane, 1);
  auto frag = [&](const uint4 (&x)[3][4][32], int kk) {
    const int l = kk & 1 ? slot1 : slot0;
    return B3{x[0][kk][l], x[1][kk][l], x[2][kk][l]};
  };
  auto frag1 = [&](const uint4 (&x)[3][32]) { return B3{x[0][slot0], x[1][slot0], x[2][slot0]}; };
  uint32_t vh[4], vl[4];      // values: bf16 as they are, fp16 as two
  auto values = [&](const S_t& st) {
    ldsm4t(vh, &st.v[8 * (m >> 1) + l8][16 * warp + 8 * (m & 1)]);
    if constexpr (kHalfIn) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&vh[i]));
        vh[i] = two(f.x, f.y);
        vl[i] = two(f.x - low(vh[i]), f.y - high(vh[i]));
      }
    }
  };
  // the values' products with two operands of two tiles each, the small ones first
  auto mma_v2 = [&](Tiles& x, Tiles& y, const B3& b, const B3& d) {
    mma_new(x[0], vh, b.lo.x, b.lo.y), mma_new(x[1], vh, b.lo.z, b.lo.w), mma_new(y[0], vh, d.lo.x, d.lo.y), mma_new(y[1], vh, d.lo.z, d.lo.w);
    if constexpr (kHalfIn) mma(x[0], vl, b.mid.x, b.mid.y), mma(x[1], vl, b.mid.z, b.mid.w), mma(y[0], vl, d.mid.x, d.mid.y), mma(y[1], vl, d.mid.z, d.mid.w);
    mma(x[0], vh, b.mid.x, b.mid.y), mma(x[1], vh, b.mid.z, b.mid.w), mma(y[0], vh, d.mid.x, d.mid.y), mma(y[1], vh, d.mid.z, d.mid.w);
    if constexpr (kHalfIn) mma(x[0], vl, b.hi.x, b.hi.y), mma(x[1], vl, b.hi.z, b.hi.w), mma(y[0], vl, d.hi.x, d.hi.y), mma(y[1], vl, d.hi.z, d.hi.w);
    mma(x[0], vh, b.hi.x, b.hi.y), mma(x[1], vh, b.hi.z, b.hi.w), mma(y[0], vh, d.hi.x, d.hi.y), mma(y[1], vh, d.hi.z, d.hi.w);
  };
  auto mma_v = [&](Tiles& x, Tiles& s, const B3& b) {     // with one, the leading products in x
    mma_new(s[0], vh, b.lo.x, b.lo.y), mma_new(s[1], vh, b.lo.z, b.lo.w);
    mma_new(x[0], vh, b.hi.x, b.hi.y), mma_new(x[1], vh, b.hi.z, b.hi.w);
    if constexpr (kHalfIn) mma(s[0], vl, b.mid.x, b.mid.y), mma(s[1], vl, b.mid.z, b.mid.w);
    mma(s[0], vh, b.mid.x, b.mid.y), mma(s[1], vh, b.mid.z, b.mid.w);
    if constexpr (kHalfIn) mma(s[0], vl, b.hi.x, b.hi.y), mma(s[1], vl, b.hi.z, b.hi.w);
  };
  // the state's channels 16 kk .. + 15 at the chunk's end
  auto carry = [&](const Ops<RULE>& ops, int kk, const Tiles& z) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int j = 2 * kk + t;
      const float2 hi = *reinterpret_cast<const float2*>(&ops.f_end[0][8 * j + 2 * c]), lo = *reinterpret_cast<const float2*>(&ops.f_end[1][8 * j + 2 * c]);
#pragma unroll
      for (int i = 0; i < 4; ++i) S[j][i] = fmaf(S[j][i], i & 1 ? hi.y : hi.x, fmaf(S[j][i], i & 1 ? lo.y : lo.x, z[t][i]));
    }
  };
  if constexpr (RULE != kDelta) {
    if (seg > 0 && !later) {                 // the state alone, from zero
      float f = 1.f, f_lo = 0.f;             // threads 0 .. 63: the product of a channel's decays
#pragma unroll
      for (int q = 0; q < kStages - 1; ++q) fetch(q, q, std::true_type{});
      int at = 0;
#pragma unroll 1
      for (int q = 0; q < n_chunks; ++q) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();
        const S_t& st = sm.stages[at];
        at = at == kStages - 1 ? 0 : at + 1;
        fetch(q + kStages - 1, at == kStages - 1 ? 0 : at + 1, std::true_type{});
        values(st);
        Tiles z0, z1, z2, z3;
        mma_v2(z0, z1, frag(st.ops.k, 0), frag(st.ops.k, 1));
        mma_v2(z2, z3, frag(st.ops.k, 2), frag(st.ops.k, 3));
        if (threadIdx.x < kDK) {
          const float g = st.ops.f_end[0][threadIdx.x], p = f * g;
          f_lo = fmaf(f_lo, g, fmaf(f, st.ops.f_end[1][threadIdx.x], fmaf(f, g, -p)));
          f = p;
        }
        carry(st.ops, 0, z0), carry(st.ops, 1, z1), carry(st.ops, 2, z2), carry(st.ops, 3, z3);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      float* end = end_of(seg);
      leave_end(end);
      if (threadIdx.x < kDK) end[kChainNT * 32 + threadIdx.x] = f, end[kChainNT * 32 + kDK + threadIdx.x] = f_lo;
      return;
    }
  }
  Split a[4];          // the state's parts (delta rule)
  auto step = [&](const Ops<RULE>& ops, int kk, const Tiles& z) {
    carry(ops, kk, z);
    split_tiles(a[kk], S[2 * kk], S[2 * kk + 1]);
  };
  if constexpr (RULE == kDelta) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) split_tiles(a[kk], S[2 * kk], S[2 * kk + 1]);
  }
#pragma unroll
  for (int q = 0; q < kStages - 1; ++q) fetch(q, q, std::false_type{});
  float* out = op + 2 * c * o_tok;
  int at = 0;
#pragma unroll 1
  for (int q = 0; q < n_chunks; ++q) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    const S_t& st = sm.stages[at];
    const Ops<RULE>& ops = st.ops;
    at = at == kStages - 1 ? 0 : at + 1;
    const int next = at == kStages - 1 ? 0 : at + 1;
    values(st);
    Tiles o, x, y, s, t;
    if constexpr (RULE == kDelta) {
      Tiles w, y0, s0, t0, v;
      mma6x2(w, y0, s0, t0, a[0], frag(ops.fk, 0), a[1], frag(ops.fk, 1));
      Tiles x1, y1, s1, t1;
      mma6x2(x1, y1, s1, t1, a[2], frag(ops.fk, 2), a[3], frag(ops.fk, 3));
      // v as accumulator tiles: times the identity
      const uint32_t one = (2 * c == r ? 0x3f80u : 0u) | (2 * c + 1 == r ? 0x3f800000u : 0u);
      mma_new(v[0], vh, one, 0u), mma_new(v[1], vh, 0u, one);
      if constexpr (kHalfIn) mma(v[0], vl, one, 0u), mma(v[1], vl, 0u, one);
      add(w, y0), add(s0, t0);
      mma6x2(o, y, s, t, a[0], frag(ops.q, 0), a[1], frag(ops.q, 1));
      fetch(q + kStages - 1, next, std::false_type{});
      add(x1, y1), add(s0, s1), add(s0, t1), add(w, x1), add(w, s0);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[g][i] -= w[g][i];
      }
      Split u;
      split_tiles(u, v[0], v[1]);
      mma6(v, s1, t1, u, frag1(ops.m));
      add(o, y), add(s, t);
      Tiles x2, y2, s2, t2;
      mma6x2(x2, y2, s2, t2, a[2], frag(ops.q, 2), a[3], frag(ops.q, 3));
      add(s1, t1), add(v, s1);
      split_tiles(u, v[0], v[1]);
      mma6x2(x1, y1, s1, t1, u, frag(ops.k, 0), u, frag(ops.k, 1));
      add(x2, y2), add(s, s2), add(s, t2);
      mma6x2(x, y, s0, t0, u, frag(ops.k, 2), u, frag1(ops.p));
      add(s1, x1), add(t1, y1);
      step(ops, 0, s1);
      mma6(x1, s2, t2, u, frag(ops.k, 3));
      step(ops, 1, t1);
      add(o, x2), add(s, t0);
      add(s0, x);
      step(ops, 2, s0);
      add(o, y);
      add(s2, t2), add(s2, x1);
      step(ops, 3, s2);
      add(o, s);
    } else {
      // channels in two halves: a half's parts of the state live for its products only, so that three CTAs fit an SM
      Tiles z0, z1, pv, ps;
      mma_v(pv, ps, frag1(ops.p));
#pragma unroll
      for (int kk = 0; kk < 4; kk += 2) {
        Split a0, a1;
        split_tiles(a0, S[2 * kk], S[2 * kk + 1]);
        split_tiles(a1, S[2 * kk + 2], S[2 * kk + 3]);
        mma_v2(z0, z1, frag(ops.k, kk), frag(ops.k, kk + 1));
        mma6x2(x, y, s, t, a0, frag(ops.q, kk), a1, frag(ops.q, kk + 1));
        if (kk == 0) fetch(q + kStages - 1, next, std::false_type{});
        carry(ops, kk, z0), carry(ops, kk + 1, z1);
        add(x, y), add(ps, s), add(ps, t);
        if (kk == 0) {
          add(x, pv);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int i = 0; i < 4; ++i) o[g][i] = x[g][i];
          }
        } else {
          add(x, ps), add(o, x);
        }
      }
    }
    const int n = n_tok - q * kTok;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if ((i >> 1 ? in1 : in0) && 8 * g + 2 * c + (i & 1) < n) out[(8 * g + (i & 1)) * o_tok + 8 * (i >> 1)] = o[g][i];
      }
    }
    out += kTok * o_tok;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (seg < last_seg) {
    if (seg == 0) leave_end(end_of(0));
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = 8 * j + 2 * c + (i & 1);
      if (e < dk && (i >> 1 ? in1 : in0)) sp[static_cast<int64_t>(e) * dv + 8 * (i >> 1)] = S[j][i];
    }
  }
}

// ---- host ---------------------------------------------------------------------------------------------------------------------------
size_t ops_bytes(int rule) { return (rule == kDelta ? sizeof(Ops<kDelta>) : sizeof(Ops<kGated>)) + sizeof(int); }
// Slots of segments' ends: a sequence of n chunks has (n - 1) / seg segments beyond its first.
int64_t slots_bound(int n_chunks, int seg) { return n_chunks / seg; }
int64_t chunk_bound(int n_tok, int n_seqs) { return static_cast<int64_t>(n_tok) / kTok + n_seqs; }

template <int RULE, typename T>
int launch_split(SplitArgs& A, void* workspace, size_t bytes, cudaStream_t stream, const char* name) {
  auto wide = [](const void* p, int64_t stride, int n) { return reinterpret_cast<uintptr_t>(p) % (2 * n) == 0 && stride % n == 0; };
  A.vec_qk = wide(A.q, A.stride, 8) && wide(A.k, A.stride, 8) && A.dk % 8 == 0;
  A.vec_a = A.a && wide(A.a, A.a_stride, 8) && A.dk % 8 == 0;
  A.vec_c = A.bias && wide(A.bias, 8, 8) && (RULE == kDelta || wide(A.rate, 8, 8)) && A.dk % 8 == 0;
  A.vec_v = wide(A.v, A.stride, 8) && A.dv % 8 == 0 ? 8 : wide(A.v, A.stride, 4) && A.dv % 4 == 0 ? 4 : 1;
  const size_t per_head = static_cast<size_t>(A.n_chunks) * ops_bytes(RULE);
  const int most = static_cast<int>(std::min<size_t>(bytes / per_head, static_cast<size_t>(A.H)));
  if (most <= 0) return fail(B200_EINVAL, "%s: workspace of %zu bytes, one head takes %zu", name, bytes, per_head);
  constexpr size_t smem = sizeof(Chain<RULE, T>);
  static_assert(kStages == 3 && sizeof(Prep<RULE>) <= 48 * 1024 && smem <= static_cast<size_t>(kMaxSmem));
  // segments: three CTAs per SM (168 registers, a few words spilled); in one piece the walk is a lone warp's latency
  auto chain = RULE != kDelta && A.seg > 0 ? split_chain_kernel<RULE, T, RULE == kDelta ? 2 : 3> : split_chain_kernel<RULE, T, 2>;
  static std::atomic<uint64_t> ready{0};      // a bit per device: the limit is always the same, a call need not set it again
  int device = 0;
  cudaGetDevice(&device);
  if (device >= 64 || !(ready.load(std::memory_order_acquire) >> device & 1)) {
    cudaFuncSetAttribute(split_chain_kernel<RULE, T, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (RULE != kDelta) cudaFuncSetAttribute(split_chain_kernel<RULE, T, RULE == kDelta ? 2 : 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (device < 64) ready.fetch_or(1ull << device, std::memory_order_release);
  }
  for (A.h0 = 0; A.h0 < A.H; A.h0 += most) {
    A.heads = std::min(most, A.H - A.h0);
    A.ops = static_cast<unsigned char*>(workspace);
    A.wild = reinterpret_cast<int*>(A.ops + static_cast<size_t>(A.n_chunks) * A.heads * sizeof(Ops<RULE>));
    split_prepare_kernel<RULE, T><<<dim3(A.n_chunks, A.heads), 128, sizeof(Prep<RULE>), stream>>>(A);
    if (int rc = check_launch(name)) return rc;
    const int extra = A.seg > 0 ? static_cast<int>(slots_bound(A.n_chunks, A.seg)) : 0, blocks = (A.dv + kCols - 1) / kCols;
    chain<<<dim3(A.n_seqs + extra, A.heads, blocks), kChainNT, smem, stream>>>(A, false);
    if (int rc = check_launch(name)) return rc;
    if (extra > 0) {
      chain<<<dim3(extra, A.heads, blocks), kChainNT, smem, stream>>>(A, true);
      if (int rc = check_launch(name)) return rc;
    }
  }
  return 0;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int b200_split_scan_supported(int dk, int dtype) { return dk > 0 && dk <= kDK && (dtype == B200_DTYPE_F16 || dtype == B200_DTYPE_BF16); }

size_t b200_split_scan_workspace(int rule, int n_tok, int n_seqs, int heads) {
  if (n_tok < 0 || n_seqs < 0 || heads < 0) return 0;
  return static_cast<size_t>(chunk_bound(n_tok, n_seqs)) * heads * ops_bytes(rule == 1 ? kDelta : kGated);
}

size_t b200_split_scan_ends(int segment, int n_tok, int n_seqs, int heads, int dv) {
  if (segment <= 0 || n_tok < 0 || n_seqs < 0 || heads < 0 || dv < 0) return 0;
  return static_cast<size_t>(slots_bound(static_cast<int>(chunk_bound(n_tok, n_seqs)), segment)) * heads * ((dv + kCols - 1) / kCols) * kEnd * sizeof(float);
}

int b200_split_scan(int rule, float* o_raw, const void* q, const void* k, const void* v, int64_t in_stride, const void* beta_logit,
                    int64_t beta_stride, const void* a_logit, int64_t a_stride, const void* bias, const void* rate, const float* decay,
                    int per_channel, float* state, const int32_t* seqs, int n_seqs, int n_tok, int H, int G, int dk, int dv,
                    float unit_eps, float scale, void* workspace, size_t workspace_bytes, int dtype, void* stream) {
  return b200_split_scan_ext(rule, o_raw, q, k, v, in_stride, beta_logit, beta_stride, a_logit, a_stride, bias, rate, decay, per_channel, state,
                             seqs, n_seqs, n_tok, H, G, dk, dv, unit_eps, scale, workspace, workspace_bytes, 0, nullptr, 0, dtype, stream);
}

int b200_split_scan_ext(int rule, float* o_raw, const void* q, const void* k, const void* v, int64_t in_stride, const void* beta_logit,
                        int64_t beta_stride, const void* a_logit, int64_t a_stride, const void* bias, const void* rate, const float* decay,
                        int per_channel, float* state, const int32_t* seqs, int n_seqs, int n_tok, int H, int G, int dk, int dv,
                        float unit_eps, float scale, void* workspace, size_t workspace_bytes, int segment, float* ends, size_t ends_bytes,
                        int dtype, void* stream) {
  const char* name = "b200_split_scan";
  if (rule < 0 || rule > 2 || n_seqs < 0 || n_tok < 0 || H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0) return fail(B200_EINVAL, "%s: bad sizes", name);
  if (!b200_split_scan_supported(dk, dtype)) return fail(B200_ESHAPE, "%s: key size %d or dtype %d not served", name, dk, dtype);
  if (n_seqs == 0) return 0;
  const bool missing = rule == kRetention ? !decay : !bias || !rate || (rule == kDelta && (!beta_logit || !a_logit));
  if (!o_raw || !q || !k || !v || !state || !seqs || !workspace || missing) return fail(B200_EINVAL, "%s: null pointer", name);
  if (!aligned16(workspace)) return fail(B200_EINVAL, "%s: workspace is not 16-byte aligned", name);
  if (segment < 0 || (segment > 0 && rule == kDelta)) return fail(B200_EINVAL, "%s: segments of %d chunks for rule %d", name, segment, rule);
  if (segment > 0 && (!ends || !aligned16(ends) || ends_bytes < b200_split_scan_ends(segment, n_tok, n_seqs, H, dv)))
    return fail(B200_EINVAL, "%s: no room for the ends of segments", name);
  SplitArgs A{};
  A.o = o_raw, A.q = q, A.k = k, A.v = v, A.stride = in_stride;
  A.beta = beta_logit, A.beta_stride = beta_stride, A.a = a_logit, A.a_stride = a_stride;
  A.bias = bias, A.rate = rate, A.decay = decay, A.per_channel = per_channel;
  A.state = state, A.seqs = reinterpret_cast<const SplitSeq*>(seqs);
  A.n_seqs = n_seqs, A.n_chunks = static_cast<int>(chunk_bound(n_tok, n_seqs));
  A.H = H, A.G = G, A.dk = dk, A.dv = dv, A.unit_eps = unit_eps, A.scale = scale;
  A.seg = segment, A.ends = ends;
  auto st = static_cast<cudaStream_t>(stream);
  auto go = [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if (rule == kGated) return launch_split<kGated, T>(A, workspace, workspace_bytes, st, name);
    if (rule == kDelta) return launch_split<kDelta, T>(A, workspace, workspace_bytes, st, name);
    return launch_split<kRetention, T>(A, workspace, workspace_bytes, st, name);
  };
  return dtype == B200_DTYPE_F16 ? go(static_cast<__half*>(nullptr)) : go(static_cast<__nv_bfloat16*>(nullptr));
}

}  // extern "C"
