// Sequence mixers and feed-forward pieces for decoder designs that keep an fp32 residual stream and run ragged
// batches (prompt portions beside single decoded tokens, packed token-major):
//
//   biased paged attention     causal softmax attention of packed query rows over the paged cache with a learned
//                              bias per (distance bucket, head), a per-position query temperature and a per-head
//                              sigmoid output gate
//   gated linear recurrence    S_t = diag(f_t) S_(t-1) + (1 - f_t) v_t^T, o_t = S_t^T q_t with the state in fp32,
//                              carried per sequence in a slot pool (kernel: b200_column_scan.cu)
//   sigmoid top-k routing, grouped linear for expert-sorted rows
// (norms, residual updates, activations and what moves rows to experts and back: b200_row_ops.cu)
//
// Every constant of a design (eps, multipliers, temperatures, limits, table sizes) is a parameter.  Scores, softmax,
// norms, gates of the recurrence, the state and the residual are fp32 whatever the storage dtype T is.  Summation
// orders of the fp32 attention and of the recurrence depend only on a token's own position and sizes, never on how a batch was
// cut, so a position's result does not change with its neighbours in the batch.  The 16-bit attention has one order for launches
// of up to 16 rows per tile (decoded tokens: key ranges at fixed multiples) and one for longer tiles; which a token gets follows from
// its portion and, where the prompt portions of a step share the launch, from those: rounding level.
#include <algorithm>
#include <type_traits>

#include "../../include/b200_mixers.h"
#include "b200_column_scan.cuh"
#include "b200_common.cuh"
#include "b200_decode_rows.cuh"

namespace b200 {

// this file is a shared library of its own: it carries its own error buffer
char* last_error_buf() {
  static thread_local char buf[kErrBufLen] = {0};
  return buf;
}

namespace {

template <typename F>
int mixer_by_dtype(int dtype, const char* name, F&& f) {
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

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }

// ---- biased paged attention over packed query rows ----------------------------------------------------------------
// A CTA serves up to QT consecutive tokens of ONE sequence and one kv head: QT * (H / G) query rows.  Keys are
// walked in tiles of 32 from position 0 (tile borders are fixed in the sequence, so the online-softmax order of a
// position does not depend on how the prompt was cut).  K and V tiles sit in shared memory as fp32; a warp owns RW
// rows, lane j scores key j of the tile, then the lanes split the value columns.
struct AttnTile {
  int tok0;   // first packed row of the tile
  int count;  // tokens in the tile (<= QT)
  int seq;    // row of the block table
};

constexpr int kAttnWarps = 8;
constexpr int kKeyTile = 32;

template <typename T, int RW, int DVL, int NCH>
__global__ void __launch_bounds__(kAttnWarps * 32)
biased_paged_attn_kernel(T* __restrict__ out, const T* __restrict__ q, int64_t q_stride, const T* __restrict__ gate,
                         int64_t gate_stride, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                         const int32_t* __restrict__ block_tables, int table_stride, const AttnTile* __restrict__ tiles,
                         const int32_t* __restrict__ tok_pos, const float* __restrict__ bias_lut, int lut_len,
                         float scale, float temp_coef, int temp_every, int H, int G, int dk, int dv, int block_size) {
  // NCH > 0: K / V rows are fetched as 16-byte chunks, NCH per thread, into registers one key tile AHEAD of the
  // tile being computed (needs dk and dv to be multiples of 16 bytes).  NCH == 0: element-wise loads, any sizes.
  extern __shared__ __align__(16) float smem[];
  const int dkp = (dk + 3) & ~3;            // padded row length of K / q rows (multiple of 4 floats)
  const int ks = dkp + 4;                   // K row stride: 16-byte aligned and conflict-free for 128-bit reads
  const int rep = H / G;
  const AttnTile tile = tiles[blockIdx.x];
  const int g = blockIdx.y;
  const int n_rows = tile.count * rep;
  float* k_s = smem;                        // [32][ks]
  float* v_s = k_s + kKeyTile * ks;         // [32][dv]
  float* q_s = v_s + kKeyTile * dv;         // [rows][dkp]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // query rows -> shared memory (fp32, zero padded)
  for (int i = threadIdx.x; i < kAttnWarps * RW * dkp; i += blockDim.x) {
    const int r = i / dkp, d = i - r * dkp;
    const int t = r / rep, hh = g * rep + (r - t * rep);
    q_s[i] = (r < n_rows && d < dk) ? Cvt<T>::to_f32(q[(tile.tok0 + t) * q_stride + hh * dk + d]) : 0.f;
  }
  const int pos_last = tok_pos[tile.tok0 + tile.count - 1];
  const int32_t* table = block_tables + static_cast<int64_t>(tile.seq) * table_stride;

  // per-row state of this warp's rows
  float m[RW], l[RW], acc[RW][DVL], qmul[RW];
  int pos[RW], head[RW];
  bool live[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const int row = warp * RW + r;
    live[r] = row < n_rows;
    const int t = live[r] ? row / rep : 0;
    head[r] = g * rep + (live[r] ? row - t * rep : 0);
    pos[r] = live[r] ? tok_pos[tile.tok0 + t] : -1;
    const float steps = static_cast<float>((pos[r] + 1) / max(temp_every, 1));
    qmul[r] = scale * (1.0f + temp_coef * logf(steps + 1.0f));
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int c = 0; c < DVL; ++c) acc[r][c] = 0.f;
  }

  constexpr int VN = 16 / sizeof(T);
  constexpr int NR = NCH > 0 ? NCH : 1;
  const int kc = dk / VN, vc = dv / VN;               // chunks per K / V row
  const int n_chunks = kKeyTile * (kc + vc);
  int4 regs[NR];
  const int bs_shift = (block_size & (block_size - 1)) == 0 ? __ffs(block_size) - 1 : -1;
  // the chunks a thread moves are the same for every key tile: (is V, key within the tile, first element) once
  int ch_j[NR], ch_e[NR];
  bool ch_v[NR], ch_ok[NR];
#pragma unroll
  for (int u = 0; u < NR; ++u) {
    const int c = threadIdx.x + u * kAttnWarps * 32;
    ch_ok[u] = NCH > 0 && c < n_chunks;
    ch_v[u] = c >= kKeyTile * kc;
    const int cc = ch_v[u] ? c - kKeyTile * kc : c;
    const int per = max(ch_v[u] ? vc : kc, 1);
    ch_j[u] = cc / per;
    ch_e[u] = (cc - ch_j[u] * per) * VN;
  }
  auto prefetch = [&](int j0) {
    const int n_keys = min(kKeyTile, pos_last + 1 - j0);
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      regs[u] = make_int4(0, 0, 0, 0);
      if (ch_ok[u] && ch_j[u] < n_keys) {
        const int key = j0 + ch_j[u];
        const int bi = bs_shift >= 0 ? key >> bs_shift : key / block_size;   // pages are a power of two as a rule
        const int64_t row = (static_cast<int64_t>(table[bi]) * G + g) * block_size + (key - bi * block_size);
        regs[u] = *reinterpret_cast<const int4*>(ch_v[u] ? v_pool + row * dv + ch_e[u] : k_pool + row * dk + ch_e[u]);
      }
    }
  };
  auto commit = [&]() {
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      if (ch_ok[u]) {
        const T* el = reinterpret_cast<const T*>(&regs[u]);
        float* dst = ch_v[u] ? v_s + ch_j[u] * dv + ch_e[u] : k_s + ch_j[u] * ks + ch_e[u];
        if constexpr (VN == 8) {
          *reinterpret_cast<float4*>(dst) = make_float4(Cvt<T>::to_f32(el[0]), Cvt<T>::to_f32(el[1]), Cvt<T>::to_f32(el[2]), Cvt<T>::to_f32(el[3]));
          *reinterpret_cast<float4*>(dst + 4) = make_float4(Cvt<T>::to_f32(el[4]), Cvt<T>::to_f32(el[5]), Cvt<T>::to_f32(el[6]), Cvt<T>::to_f32(el[7]));
        } else {
          *reinterpret_cast<float4*>(dst) = make_float4(Cvt<T>::to_f32(el[0]), Cvt<T>::to_f32(el[1]), Cvt<T>::to_f32(el[2]), Cvt<T>::to_f32(el[3]));
        }
      }
    }
  };
  if constexpr (NCH > 0) prefetch(0);

  for (int j0 = 0; j0 <= pos_last; j0 += kKeyTile) {
    __syncthreads();  // previous tile fully consumed (and q_s written, on the first pass)
    const int n_keys = min(kKeyTile, pos_last + 1 - j0);
    if constexpr (NCH > 0) {
      commit();
    } else {
      for (int i = threadIdx.x; i < kKeyTile * dkp; i += blockDim.x) {
        const int j = i / dkp, d = i - j * dkp;
        float f = 0.f;
        if (j < n_keys && d < dk) {
          const int key = j0 + j;
          const int64_t blk = table[key / block_size];
          f = Cvt<T>::to_f32(k_pool[((blk * G + g) * block_size + key % block_size) * dk + d]);
        }
        k_s[j * ks + d] = f;
      }
      for (int i = threadIdx.x; i < kKeyTile * dv; i += blockDim.x) {
        const int j = i / dv, c = i - j * dv;
        float f = 0.f;
        if (j < n_keys) {
          const int key = j0 + j;
          const int64_t blk = table[key / block_size];
          f = Cvt<T>::to_f32(v_pool[((blk * G + g) * block_size + key % block_size) * dv + c]);
        }
        v_s[i] = f;
      }
    }
    __syncthreads();
    if constexpr (NCH > 0) {
      if (j0 + kKeyTile <= pos_last) prefetch(j0 + kKeyTile);
    }

    if (warp * RW < n_rows) {   // warps without a live row only help with the loads and barriers
    // scores: lane = key of the tile
    float s[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) s[r] = 0.f;
    const float4* kr = reinterpret_cast<const float4*>(k_s + lane * ks);
    for (int d4 = 0; d4 < dkp / 4; ++d4) {
      const float4 kv = kr[d4];
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const float4 qv = reinterpret_cast<const float4*>(q_s + (warp * RW + r) * dkp)[d4];  // broadcast read
        s[r] = fmaf(qv.x, kv.x, s[r]);
        s[r] = fmaf(qv.y, kv.y, s[r]);
        s[r] = fmaf(qv.z, kv.z, s[r]);
        s[r] = fmaf(qv.w, kv.w, s[r]);
      }
    }
    float p[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const int key = j0 + lane;
      const bool seen = live[r] && key <= pos[r];
      const bool any = live[r] && j0 <= pos[r];  // warp-uniform
      float sc = -INFINITY;
      if (seen) {
        const int dist = min(pos[r] - key, lut_len - 1);
        sc = s[r] * qmul[r] + bias_lut[head[r] * lut_len + dist];
      }
      p[r] = 0.f;
      if (any) {
        const float m_new = fmaxf(m[r], warp_max(sc));
        const float corr = expf(m[r] - m_new);
        p[r] = seen ? expf(sc - m_new) : 0.f;
        l[r] = l[r] * corr + warp_sum(p[r]);
        m[r] = m_new;
#pragma unroll
        for (int c = 0; c < DVL; ++c) acc[r][c] *= corr;
      }
    }
    // values: lane = column (plus 32 c)
    for (int j = 0; j < n_keys; ++j) {
      float vv[DVL];
#pragma unroll
      for (int c = 0; c < DVL; ++c) {
        const int col = lane + 32 * c;
        vv[c] = col < dv ? v_s[j * dv + col] : 0.f;
      }
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const float pj = __shfl_sync(0xffffffffu, p[r], j);
#pragma unroll
        for (int c = 0; c < DVL; ++c) acc[r][c] = fmaf(pj, vv[c], acc[r][c]);
      }
    }
    }
  }

#pragma unroll
  for (int r = 0; r < RW; ++r) {
    if (!live[r]) continue;
    const int row = warp * RW + r;
    const int t = row / rep;
    const int64_t n = tile.tok0 + t;
    const float gt = gate ? sigmoidf_(Cvt<T>::to_f32(gate[n * gate_stride + head[r]])) : 1.0f;
    const float inv = gt / l[r];
#pragma unroll
    for (int c = 0; c < DVL; ++c) {
      const int col = lane + 32 * c;
      if (col < dv) out[(n * H + head[r]) * dv + col] = Cvt<T>::from_f32(acc[r][c] * inv);
    }
  }
}

// ---- biased attention for prompt portions on the tensor cores (16-bit storage types) --------------------------------
// A CTA serves up to 64 consecutive tokens of one sequence and ONE query head; warp w owns rows 16 w .. 16 w + 15.
// Keys are walked in tiles of 64 from position 0.  K and V tiles arrive by cp.async, double buffered, and stay in
// their storage type; S = Q K^T and O += P V are mma.sync m16n8k16 with fp32 accumulators in registers, the softmax
// (scale, temperature, bias, causal mask, running max and sum) runs in fp32 on the S fragments, and only the
// weights P are rounded to the storage type as the left operand of P V.  V fragments come from ldmatrix.trans.
template <typename T>
struct Mma16;
template <>
struct Mma16<__nv_bfloat16> {
  static __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
};
template <>
struct Mma16<__half> {
  static __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
};

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src, bool valid) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  const int bytes = valid ? 16 : 0;  // fewer source bytes than 16: the rest is zero-filled
  // no memory clobber: what the next copies need may be looked up in between (commit and wait carry it)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem_src), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int kMmaRows = 64;   // query rows per CTA
constexpr int kMmaKeys = 64;   // keys per tile

// KSPLIT (tiles of at most 16 rows, i.e. decoded tokens): all four warps work on the SAME 16 rows and each takes 16
// of a tile's 64 keys; their running (max, sum, output) are merged through shared memory at the end.  With a workspace the keys are
// divided over CTAs as well, kSplitKeys at absolute multiples each (so a token's sums do not depend on its neighbours): one CTA per
// sequence and kv head left the chip to the longest sequences, 163 us for 48 sequences of up to 3000 tokens over 4 kv heads.
constexpr int kSplitKeys = 256;
constexpr int kMmaRowsSplit = 16;
template <typename T, int DV8, bool KSPLIT>
__global__ void __launch_bounds__(128)
biased_prompt_attn_mma_kernel(T* __restrict__ out, const T* __restrict__ q, int64_t q_stride, const T* __restrict__ gate,
                              int64_t gate_stride, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                              const int32_t* __restrict__ block_tables, int table_stride,
                              const AttnTile* __restrict__ tiles, const int32_t* __restrict__ tok_pos,
                              const float* __restrict__ bias_lut, int lut_len, int lut_in_smem, int q_vec, float scale,
                              float temp_coef, int temp_every, int H, int G, int dk, int dv, int block_size, float* __restrict__ ws,
                              int ws_tile) {
  // Row r of the CTA's 64 is (token r / rep, head g * rep + r % rep): the heads of a kv group share the K / V tiles.
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int dvp = DV8 * 8;
  const int ldq = dk + 8, ldv = dvp + 8;       // element strides: 16-byte multiples, conflict-free fragment reads
  T* q_s = reinterpret_cast<T*>(smem_raw);     // [64 or 16][ldq]
  constexpr int kQRows = KSPLIT ? kMmaRowsSplit : kMmaRows;
  T* k_s = q_s + kQRows * ldq;                 // 2 x [64][ldq]
  T* v_s = k_s + 2 * kMmaKeys * ldq;           // 2 x [64][ldv]
  float* lut_s = reinterpret_cast<float*>(v_s + 2 * kMmaKeys * ldv);
  const AttnTile tile = tiles[blockIdx.x];
  const int g = blockIdx.y, rep = H / G;
  const int n_rows = tile.count * rep;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int pos0 = tok_pos[tile.tok0];
  const int pos_last = pos0 + tile.count - 1;
  // key tiles of this CTA: all, or its kSplitKeys
  const bool split = KSPLIT && ws != nullptr;
  const int kt0 = split ? blockIdx.z * (kSplitKeys / kMmaKeys) : 0;
  const int kt1 = split ? min(pos_last / kMmaKeys + 1, kt0 + kSplitKeys / kMmaKeys) : pos_last / kMmaKeys + 1;
  if (kt0 >= kt1) return;
  const int32_t* table = block_tables + static_cast<int64_t>(tile.seq) * table_stride;
  if (lut_in_smem) {   // the group's heads, one after the other
    for (int i = threadIdx.x; i < rep * lut_len; i += blockDim.x) lut_s[i] = bias_lut[static_cast<int64_t>(g) * rep * lut_len + i];
  }
  const int qc = dk / 8, vc = dvp / 8;          // 16-byte chunks per row

  // Q tile (rows beyond the tile's are zero); element-wise when the rows are not 16-byte aligned
  if (q_vec) {
    for (int c = threadIdx.x; c < kQRows * qc; c += blockDim.x) {
      const int r = c / qc, e = (c - r * qc) * 8;
      const bool ok = r < n_rows;
      const int t = r / rep, hh = g * rep + (r - t * rep);
      cp_async16(q_s + r * ldq + e, ok ? q + (tile.tok0 + t) * q_stride + hh * dk + e : q, ok);
    }
  } else {
    for (int i = threadIdx.x; i < kQRows * dk; i += blockDim.x) {
      const int r = i / dk, d = i - r * dk;
      const int t = r / rep, hh = g * rep + (r - t * rep);
      q_s[r * ldq + d] = r < n_rows ? q[(tile.tok0 + t) * q_stride + hh * dk + d] : Cvt<T>::from_f32(0.f);
    }
  }
  // a thread always moves the same 16-byte column of the rows j = row0, row0 + step, ...: no division per chunk
  const int bs_shift = (block_size & (block_size - 1)) == 0 ? __ffs(block_size) - 1 : -1;
  const int k_step = blockDim.x / qc, k_row0 = threadIdx.x / qc, k_e = (threadIdx.x - k_row0 * qc) * 8;
  const int v_step = blockDim.x / vc, v_row0 = threadIdx.x / vc, v_e = (threadIdx.x - v_row0 * vc) * 8;
  auto pool_row = [&](int key) -> int64_t {
    const int bi = bs_shift >= 0 ? key >> bs_shift : key / block_size;
    return (static_cast<int64_t>(table[bi]) * G + g) * block_size + (key - bi * block_size);
  };
  auto load_kv = [&](int j0, int stage) {
    T* kd = k_s + stage * kMmaKeys * ldq;
    T* vd = v_s + stage * kMmaKeys * ldv;
    // four rows at a time: their look-ups overlap, and none waits between two copies
    auto rows = [&](T* dst, const T* pool, int ld, int width, int row0, int step, int e, bool col_ok) {
      if (row0 >= step) return;
      for (int j = row0; j < kMmaKeys; j += 4 * step) {
        int64_t r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int key = j0 + j + u * step;
          r[u] = col_ok && j + u * step < kMmaKeys && key <= pos_last ? pool_row(key) : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool ok = r[u] >= 0;
          if (j + u * step < kMmaKeys) cp_async16(dst + (j + u * step) * ld + e, pool + (ok ? r[u] * width + e : 0), ok);
        }
      }
    };
    rows(kd, k_pool, ldq, dk, k_row0, k_step, k_e, true);
    rows(vd, v_pool, ldv, dv, v_row0, v_step, v_e, v_e < dv);
  };
  load_kv(kt0 * kMmaKeys, 0);
  cp_async_commit();

  const int row_a = (KSPLIT ? 0 : warp * 16) + gq;       // this thread's rows: row_a and row_a + 8
  int posr[2], headr[2], tokr[2];
  const float* lut[2];
  float qmul[2], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = row_a + 8 * i;
    tokr[i] = r / rep;
    headr[i] = g * rep + (r - tokr[i] * rep);
    posr[i] = r < n_rows ? pos0 + tokr[i] : -1;
    lut[i] = lut_in_smem ? lut_s + (r - tokr[i] * rep) * lut_len : bias_lut + static_cast<int64_t>(headr[i]) * lut_len;
    const float steps = static_cast<float>((posr[i] + 1) / max(temp_every, 1));
    qmul[i] = scale * (1.0f + temp_coef * logf(steps + 1.0f));
  }
  const int warp_pos_max = KSPLIT ? pos_last : pos0 + min((warp * 16 + 15) / rep, tile.count - 1);
  const bool warp_live = KSPLIT || warp * 16 < n_rows;
  constexpr int NT = KSPLIT ? 2 : 8;                     // 8-key n-tiles of a key tile this warp scores
  const int nt0 = KSPLIT ? 2 * warp : 0;
  float o[DV8][4];
#pragma unroll
  for (int n = 0; n < DV8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

  for (int it = kt0; it < kt1; ++it) {
    const int stage = (it - kt0) & 1;
    if (it + 1 < kt1) {
      load_kv((it + 1) * kMmaKeys, stage ^ 1);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const int j0 = it * kMmaKeys;
    if (warp_live && j0 <= warp_pos_max) {
      const T* kt = k_s + stage * kMmaKeys * ldq;
      const T* vt = v_s + stage * kMmaKeys * ldv;
      float s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
      for (int kk = 0; kk < dk / 16; ++kk) {
        uint32_t a[4];
        const T* qa = q_s + row_a * ldq + kk * 16 + 2 * tq;
        a[0] = *reinterpret_cast<const uint32_t*>(qa);
        a[1] = *reinterpret_cast<const uint32_t*>(qa + 8 * ldq);
        a[2] = *reinterpret_cast<const uint32_t*>(qa + 8);
        a[3] = *reinterpret_cast<const uint32_t*>(qa + 8 * ldq + 8);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const T* kb = kt + ((nt0 + n) * 8 + gq) * ldq + kk * 16 + 2 * tq;
          Mma16<T>::mma(s[n], a, *reinterpret_cast<const uint32_t*>(kb), *reinterpret_cast<const uint32_t*>(kb + 8));
        }
      }
      // fp32 softmax on the fragments: element e of s[n] is (row gq + 8 (e >> 1), key 8 (nt0 + n) + 2 tq + (e & 1))
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = e >> 1;
          const int key = j0 + (nt0 + n) * 8 + 2 * tq + (e & 1);
          float sc = -INFINITY;
          if (key <= posr[i]) sc = s[n][e] * qmul[i] + lut[i][min(posr[i] - key, lut_len - 1)];
          s[n][e] = sc;
          mx[i] = fmaxf(mx[i], sc);
        }
      }
      float corr[2], msafe[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        const float m_new = fmaxf(m[i], mx[i]);
        msafe[i] = m_new == -INFINITY ? 0.f : m_new;   // a row that sees no key yet keeps weights 0, not NaN
        corr[i] = expf(m[i] - msafe[i]);
        m[i] = m_new;
      }
      float part[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float pexp = expf(s[n][e] - msafe[e >> 1]);
          s[n][e] = pexp;
          part[e >> 1] += pexp;
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) l[i] = l[i] * corr[i] + part[i];   // per-thread share of the row sum
#pragma unroll
      for (int n = 0; n < DV8; ++n) {
        o[n][0] *= corr[0];
        o[n][1] *= corr[0];
        o[n][2] *= corr[1];
        o[n][3] *= corr[1];
      }
#pragma unroll
      for (int k2 = 0; k2 < NT / 2; ++k2) {
        uint32_t a[4];
        a[0] = Mma16<T>::pack(s[2 * k2][0], s[2 * k2][1]);
        a[1] = Mma16<T>::pack(s[2 * k2][2], s[2 * k2][3]);
        a[2] = Mma16<T>::pack(s[2 * k2 + 1][0], s[2 * k2 + 1][1]);
        a[3] = Mma16<T>::pack(s[2 * k2 + 1][2], s[2 * k2 + 1][3]);
        const int key16 = (nt0 / 2 + k2) * 16;           // first key (within the tile) of this 16-key step
#pragma unroll
        for (int n = 0; n < DV8; n += 2) {
          const T* vrow = vt + (key16 + (lane & 7) + ((lane >> 3) & 1) * 8) * ldv + n * 8 + (lane >> 4) * 8;
          const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(vrow));
          uint32_t b0, b1, b2, b3;
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                       : "r"(addr));
          Mma16<T>::mma(o[n], a, b0, b1);
          Mma16<T>::mma(o[n + 1], a, b2, b3);
        }
      }
    }
    __syncthreads();   // the stage just read is the target of the load after next
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
  if constexpr (KSPLIT) {
    // merge the four warps' partial results for the 16 shared rows: every warp rescales its own to the common
    // maximum and the sums are taken warp 0, 1, 2, 3 in order; the K / V stages are free now
    float* mg = reinterpret_cast<float*>(k_s);            // [4 warps][16 rows] maxima, then [4][16] sums
    float* og = mg + 128;                                  // [4 warps][16 rows][dvp]
    if (tq == 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mg[warp * 16 + gq + 8 * i] = m[i];
        mg[64 + warp * 16 + gq + 8 * i] = l[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = gq + 8 * i;
      const float seen = fmaxf(fmaxf(mg[r], mg[16 + r]), fmaxf(mg[32 + r], mg[48 + r]));   // -inf: none of these keys
      const float mall = seen == -INFINITY ? 0.f : seen;
      const float w = expf(m[i] - mall);                  // this warp's weight in the merge
      float lsum = 0.f;
#pragma unroll
      for (int w2 = 0; w2 < 4; ++w2) lsum += mg[64 + w2 * 16 + r] * expf(mg[w2 * 16 + r] - mall);
      l[i] = lsum;
      m[i] = seen;
#pragma unroll
      for (int n = 0; n < DV8; ++n) {
        og[(warp * 16 + r) * dvp + n * 8 + 2 * tq] = o[n][2 * i] * w;
        og[(warp * 16 + r) * dvp + n * 8 + 2 * tq + 1] = o[n][2 * i + 1] * w;
      }
    }
    __syncthreads();
    if (!split && warp != 0) return;
    if (split) {     // (maximum, sum, output) of these keys, all warps: the merge kernel below reads them
      const int64_t ws_row0 = (static_cast<int64_t>(blockIdx.z) * gridDim.x + blockIdx.x) * ws_tile;
      for (int e = threadIdx.x; e < n_rows * dv; e += blockDim.x) {
        const int r = e / dv, c = e - r * dv, t = r / rep;
        float* dst = ws + ((ws_row0 + t) * H + g * rep + r - t * rep) * (dv + 2);
        dst[2 + c] = (og[r * dvp + c] + og[(16 + r) * dvp + c]) + (og[(32 + r) * dvp + c] + og[(48 + r) * dvp + c]);
      }
      if (warp == 0 && tq == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (gq + 8 * i >= n_rows) continue;
          float* dst = ws + ((ws_row0 + tokr[i]) * H + headr[i]) * (dv + 2);
          dst[0] = m[i];
          dst[1] = l[i];
        }
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = gq + 8 * i;
#pragma unroll
      for (int n = 0; n < DV8; ++n) {
        const int c = n * 8 + 2 * tq;
        o[n][2 * i] = (og[r * dvp + c] + og[(16 + r) * dvp + c]) + (og[(32 + r) * dvp + c] + og[(48 + r) * dvp + c]);
        o[n][2 * i + 1] = (og[r * dvp + c + 1] + og[(16 + r) * dvp + c + 1]) + (og[(32 + r) * dvp + c + 1] + og[(48 + r) * dvp + c + 1]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = row_a + 8 * i;
    if (r >= n_rows) continue;
    const int64_t n_tok = tile.tok0 + tokr[i];
    const int h = headr[i];
    const float gt = gate ? sigmoidf_(Cvt<T>::to_f32(gate[n_tok * gate_stride + h])) : 1.0f;
    const float inv = gt / l[i];
    T* orow = out + (n_tok * H + h) * dv;
#pragma unroll
    for (int n = 0; n < DV8; ++n) {
      const int col = n * 8 + 2 * tq;
      if (col < dv) {   // dv is a multiple of 8: col + 1 < dv as well
        orow[col] = Cvt<T>::from_f32(o[n][2 * i] * inv);
        orow[col + 1] = Cvt<T>::from_f32(o[n][2 * i + 1] * inv);
      }
    }
  }
}

// The key splits of a token and head brought together: one CTA per (tile, token of it, head), a thread per value column.
template <typename T>
__global__ void __launch_bounds__(128)
biased_split_merge_kernel(T* __restrict__ out, const float* __restrict__ ws, const T* __restrict__ gate, int64_t gate_stride,
                          const AttnTile* __restrict__ tiles, const int32_t* __restrict__ tok_pos, int H, int dv) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const AttnTile tile = tiles[blockIdx.x];
  if (static_cast<int>(blockIdx.y) >= tile.count) return;
  const int64_t n = tile.tok0 + blockIdx.y;
  const int h = blockIdx.z, c = threadIdx.x, lane = threadIdx.x & 31;
  const int splits = (tok_pos[tile.tok0] + tile.count - 1) / kSplitKeys + 1;     // as the tile's CTAs cut its keys
  const int64_t step = static_cast<int64_t>(gridDim.x) * gridDim.y * H * (dv + 2);
  const float* src = ws + ((static_cast<int64_t>(blockIdx.x) * gridDim.y + blockIdx.y) * H + h) * (dv + 2);
  float M = -INFINITY;      // a lane per split: one trip to memory for all maxima and sums
  for (int sp = lane; sp < splits; sp += 32) M = fmaxf(M, src[sp * step]);
  M = warp_max(M);
  float L = 0.f, O = 0.f;
  for (int base = 0; base < splits; base += 32) {
    const int sp = base + lane, here = min(32, splits - base);
    const float f = sp < splits ? expf(src[sp * step] - M) : 0.f;      // a row that saw none of a split's keys left -inf, 0 and 0
    const float lf = sp < splits ? src[sp * step + 1] * f : 0.f;
    L += warp_sum(lf);
#pragma unroll 8
    for (int u = 0; u < here; ++u) {
      const float fu = __shfl_sync(0xffffffffu, f, u);
      if (c < dv) O = fmaf(src[(base + u) * step + 2 + c], fu, O);
    }
  }
  if (c >= dv) return;
  // in the order of the launch without splits, whose result a row of one range repeats to the bit
  const float gt = gate ? sigmoidf_(Cvt<T>::to_f32(gate[n * gate_stride + h])) : 1.0f;
  const float inv = gt / L;
  out[(n * H + h) * dv + c] = Cvt<T>::from_f32(O * inv);
}

// ---- grouped linear for expert-sorted rows (16-bit storage) ---------------------------------------------------------
// out[r] = xs[r] . w[e]^T for the rows offsets[e] <= r < offsets[e + 1]; the offsets stay on the device, so routing
// needs no copy to the host and all experts run in one launch.  CTA = 16 rows x 256 output columns of one expert
// (each of 4 warps: 16 x 64 with mma.sync m16n8k16, fp32 accumulators); K in chunks of 64 by cp.async, two stages.
// CTAs whose row tile lies beyond their expert's rows leave at once.
constexpr int kGrpRows = 16, kGrpCols = 256, kGrpK = 64;

template <typename T>
__global__ void __launch_bounds__(128)
grouped_linear_kernel(T* __restrict__ out, const T* __restrict__ xs, const T* __restrict__ w,
                      const int32_t* __restrict__ offsets, int N, int K) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int e = blockIdx.y;
  const int row0 = offsets[e] + blockIdx.z * kGrpRows;
  const int row_end = offsets[e + 1];
  if (row0 >= row_end) return;
  const int n0 = blockIdx.x * kGrpCols;
  constexpr int ld = kGrpK + 8;
  T* x_s = reinterpret_cast<T*>(smem_raw);            // 2 x [16][ld]
  T* w_s = x_s + 2 * kGrpRows * ld;                   // 2 x [256][ld]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const T* wbase = w + static_cast<int64_t>(e) * N * K;
  auto load = [&](int kc, int stage) {
    {
      const int r = threadIdx.x >> 3, e8 = (threadIdx.x & 7) * 8;
      const bool ok = row0 + r < row_end && kc + e8 < K;
      cp_async16(x_s + (stage * kGrpRows + r) * ld + e8, ok ? xs + static_cast<int64_t>(row0 + r) * K + kc + e8 : xs, ok);
    }
#pragma unroll 4
    for (int i = 0; i < kGrpCols * 8 / 128; ++i) {
      const int c = threadIdx.x + i * 128;
      const int n = c >> 3, e8 = (c & 7) * 8;
      const bool ok = n0 + n < N && kc + e8 < K;
      cp_async16(w_s + (stage * kGrpCols + n) * ld + e8, ok ? wbase + static_cast<int64_t>(n0 + n) * K + kc + e8 : wbase, ok);
    }
  };
  float acc[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const int n_kc = (K + kGrpK - 1) / kGrpK;
  load(0, 0);
  cp_async_commit();
  for (int it = 0; it < n_kc; ++it) {
    if (it + 1 < n_kc) {
      load((it + 1) * kGrpK, (it + 1) & 1);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const T* xt = x_s + (it & 1) * kGrpRows * ld;
    const T* wt = w_s + ((it & 1) * kGrpCols + warp * 64) * ld;
#pragma unroll
    for (int kk = 0; kk < kGrpK / 16; ++kk) {
      uint32_t a[4];
      const T* xa = xt + gq * ld + kk * 16 + 2 * tq;
      a[0] = *reinterpret_cast<const uint32_t*>(xa);
      a[1] = *reinterpret_cast<const uint32_t*>(xa + 8 * ld);
      a[2] = *reinterpret_cast<const uint32_t*>(xa + 8);
      a[3] = *reinterpret_cast<const uint32_t*>(xa + 8 * ld + 8);
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const T* wb = wt + (n * 8 + gq) * ld + kk * 16 + 2 * tq;
        Mma16<T>::mma(acc[n], a, *reinterpret_cast<const uint32_t*>(wb), *reinterpret_cast<const uint32_t*>(wb + 8));
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = row0 + gq + 8 * i;
    if (r >= row_end) continue;
    T* orow = out + static_cast<int64_t>(r) * N;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int col = n0 + warp * 64 + n * 8 + 2 * tq;
      if (col < N) orow[col] = Cvt<T>::from_f32(acc[n][2 * i]);
      if (col + 1 < N) orow[col + 1] = Cvt<T>::from_f32(acc[n][2 * i + 1]);
    }
  }
}

// ---- routing ----------------------------------------------------------------------------------------------------
// One warp per token: the `top` largest logits (ties: lowest index), weight = sigmoid(logit).  NaN logits are chosen last, the lowest
// index first: the ids address experts and rows, so a token of NaNs has to have some, and its weights are NaN.
__global__ void __launch_bounds__(128)
sigmoid_topk_kernel(int32_t* __restrict__ ids, float* __restrict__ weights, const float* __restrict__ logits, int n_tok,
                    int E, int top) {
  const int tok = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (tok >= n_tok) return;
  const int lane = threadIdx.x & 31;
  const float* z = logits + static_cast<int64_t>(tok) * E;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      bool taken = false;
      for (int j = 0; j < k; ++j) taken |= ids[static_cast<int64_t>(tok) * top + j] == e;
      const float f = z[e];
      if (!taken && (f > best || (f == best && e < bi))) {
        best = f;
        bi = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    if (lane == 0) {
      if (bi == 0x7fffffff) {        // what is left is NaN
        auto taken = [&](int e) {
          for (int j = 0; j < k; ++j)
            if (ids[static_cast<int64_t>(tok) * top + j] == e) return true;
          return false;
        };
        for (bi = 0; taken(bi);) ++bi;
        best = z[bi];
      }
      ids[static_cast<int64_t>(tok) * top + k] = bi;
      weights[static_cast<int64_t>(tok) * top + k] = sigmoidf_(best);
    }
    __syncwarp();
  }
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

int b200_mixers_abi_version(void) { return B200_MIXERS_ABI_VERSION; }

const char* b200_mixers_last_error(void) { return last_error_buf(); }

int b200_biased_attn_tile_tokens(int n_tokens_in_portion, int H, int G) {
  // tokens per CTA: prompt portions fill 8 warps x 4 rows, a decoded token takes what its head group needs
  const int rep = std::max(1, H / std::max(G, 1));
  const int rows_max = kAttnWarps * 4;
  return std::max(1, std::min(n_tokens_in_portion, rows_max / std::min(rep, rows_max)));
}

int b200_biased_paged_attn(void* out, const void* q, int64_t q_stride, const void* gate, int64_t gate_stride,
                           const void* k_pool, const void* v_pool, const int32_t* block_tables, int table_stride,
                           const int32_t* tiles, int n_tiles, int max_tile_tokens, const int32_t* tok_pos,
                           const float* bias_lut, int lut_len, float scale, float temp_coef, int temp_every, int H, int G,
                           int dk, int dv, int block_size, int dtype, void* stream) {
  if (n_tiles < 0 || H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0 || dv > 256 || block_size <= 0 || lut_len <= 0 ||
      max_tile_tokens <= 0)
    return fail(B200_EINVAL, "b200_biased_paged_attn: bad sizes");
  if (n_tiles == 0) return 0;
  if (!out || !q || !k_pool || !v_pool || !block_tables || !tiles || !tok_pos || !bias_lut)
    return fail(B200_EINVAL, "b200_biased_paged_attn: null pointer");
  const int rep = H / G;
  const int rows = max_tile_tokens * rep;
  if (rows > kAttnWarps * 4) return fail(B200_ESHAPE, "b200_biased_paged_attn: %d rows per tile > %d", rows, kAttnWarps * 4);
  const int dkp = (dk + 3) & ~3;
  const int rw = rows <= kAttnWarps ? 1 : (rows <= 2 * kAttnWarps ? 2 : 4);  // rows per warp (template RW)
  const size_t smem = sizeof(float) * (static_cast<size_t>(kKeyTile) * (dkp + 4) + static_cast<size_t>(kKeyTile) * dv +
                                       static_cast<size_t>(kAttnWarps) * rw * dkp);
  if (smem > 200 * 1024) return fail(B200_ESHAPE, "b200_biased_paged_attn: head sizes %d / %d need too much shared memory", dk, dv);
  const dim3 grid(n_tiles, G);
  return mixer_by_dtype(dtype, "b200_biased_paged_attn", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    auto launch = [&](auto kern) {
      if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
      kern<<<grid, kAttnWarps * 32, smem, static_cast<cudaStream_t>(stream)>>>(
          static_cast<T*>(out), static_cast<const T*>(q), q_stride, static_cast<const T*>(gate), gate_stride,
          static_cast<const T*>(k_pool), static_cast<const T*>(v_pool), block_tables, table_stride,
          reinterpret_cast<const AttnTile*>(tiles), tok_pos, bias_lut, lut_len, scale, temp_coef, temp_every, H, G, dk, dv,
          block_size);
    };
    const int dvl = (dv + 31) / 32;
    // 16-byte chunk loads with a one-tile register prefetch when rows are multiples of 16 bytes and a tile's chunks
    // fit 4 (or 8) per thread; element-wise loads otherwise
    constexpr int VN = 16 / static_cast<int>(sizeof(T));
    const bool vec = dk % VN == 0 && dv % VN == 0 && aligned16(k_pool) && aligned16(v_pool);
    const int per_thread = vec ? (kKeyTile * (dk / VN + dv / VN) + kAttnWarps * 32 - 1) / (kAttnWarps * 32) : 0;
    const int nch = !vec || per_thread > 8 ? 0 : (per_thread <= 4 ? 4 : 8);
#define B200_ATTN_DV(RW_, NCH_)                                              \
  if (dvl <= 1) launch(biased_paged_attn_kernel<T, RW_, 1, NCH_>);           \
  else if (dvl <= 2) launch(biased_paged_attn_kernel<T, RW_, 2, NCH_>);      \
  else if (dvl <= 4) launch(biased_paged_attn_kernel<T, RW_, 4, NCH_>);      \
  else launch(biased_paged_attn_kernel<T, RW_, 8, NCH_>);
#define B200_ATTN_CASE(RW_)                                                  \
  if (nch == 4) { B200_ATTN_DV(RW_, 4) }                                     \
  else if (nch == 8) { B200_ATTN_DV(RW_, 8) }                                \
  else { B200_ATTN_DV(RW_, 0) }
    if (rw <= 1) { B200_ATTN_CASE(1) }
    else if (rw <= 2) { B200_ATTN_CASE(2) }
    else { B200_ATTN_CASE(4) }
#undef B200_ATTN_CASE
#undef B200_ATTN_DV
    return check_launch("b200_biased_paged_attn");
  });
}

int b200_biased_prompt_attn_tile_tokens(int H, int G) { return std::max(1, kMmaRows / std::max(1, H / std::max(G, 1))); }

int b200_biased_prompt_attn_supported(int dk, int dv, int dtype) {
  return (dtype == B200_DTYPE_BF16 || dtype == B200_DTYPE_F16) && dk > 0 && dk % 16 == 0 && dk <= 256 && dv > 0 &&
         dv % 8 == 0 && dv <= 128;
}

int b200_biased_prompt_attn(void* out, const void* q, int64_t q_stride, const void* gate, int64_t gate_stride,
                            const void* k_pool, const void* v_pool, const int32_t* block_tables, int table_stride,
                            const int32_t* tiles, int n_tiles, int max_tile_tokens, const int32_t* tok_pos, const float* bias_lut,
                            int lut_len, float scale, float temp_coef, int temp_every, int H, int G, int dk, int dv,
                            int block_size, int dtype, void* stream) {
  return b200_biased_prompt_attn_ext(out, q, q_stride, gate, gate_stride, k_pool, v_pool, block_tables, table_stride, tiles, n_tiles,
                                     max_tile_tokens, tok_pos, bias_lut, lut_len, scale, temp_coef, temp_every, H, G, dk, dv, block_size,
                                     0, nullptr, dtype, stream);
}

int b200_biased_attn_split_keys(void) { return kSplitKeys; }

int b200_biased_prompt_attn_ext(void* out, const void* q, int64_t q_stride, const void* gate, int64_t gate_stride,
                            const void* k_pool, const void* v_pool, const int32_t* block_tables, int table_stride,
                            const int32_t* tiles, int n_tiles, int max_tile_tokens, const int32_t* tok_pos, const float* bias_lut,
                            int lut_len, float scale, float temp_coef, int temp_every, int H, int G, int dk, int dv,
                            int block_size, int max_context, float* workspace, int dtype, void* stream) {
  if (n_tiles < 0 || H <= 0 || G <= 0 || H % G || block_size <= 0 || lut_len <= 0)
    return fail(B200_EINVAL, "b200_biased_prompt_attn: bad sizes");
  if (!b200_biased_prompt_attn_supported(dk, dv, dtype))
    return fail(B200_ESHAPE, "b200_biased_prompt_attn: needs a 16-bit dtype, dk %% 16 == 0 (<= 256), dv %% 8 == 0 (<= 128)");
  if (n_tiles == 0) return 0;
  if (!out || !q || !k_pool || !v_pool || !block_tables || !tiles || !tok_pos || !bias_lut)
    return fail(B200_EINVAL, "b200_biased_prompt_attn: null pointer");
  if (!aligned16(k_pool) || !aligned16(v_pool))
    return fail(B200_ESHAPE, "b200_biased_prompt_attn: pools must be 16-byte aligned");
  const int q_vec = aligned16(q) && (q_stride * 2) % 16 == 0;
  const int dv8 = dv <= 32 ? 4 : (dv <= 64 ? 8 : 16);
  const int rep = H / G;
  if (rep > kMmaRows) return fail(B200_ESHAPE, "b200_biased_prompt_attn: %d heads per kv head > %d", rep, kMmaRows);
  // tiles of at most 16 rows (decoded tokens): the four warps split the keys instead of the rows, and with a workspace CTAs do too
  const bool ksplit = max_tile_tokens > 0 && max_tile_tokens * rep <= kMmaRowsSplit;
  const int n_splits = ksplit && workspace && max_context > kSplitKeys ? (max_context + kSplitKeys - 1) / kSplitKeys : 1;
  const size_t tiles_bytes = 2u * (static_cast<size_t>(dk + 8) * ((ksplit ? kMmaRowsSplit : kMmaRows) + 2u * kMmaKeys) + 2u * kMmaKeys * (dv8 * 8 + 8));
  // the group's bias tables go to shared memory when they are small enough to leave room for two CTAs per SM
  const size_t lut_bytes = static_cast<size_t>(rep) * lut_len * 4;
  const int lut_in_smem = lut_bytes <= 20 * 1024;
  const size_t smem = tiles_bytes + (lut_in_smem ? lut_bytes : 0);
  const dim3 grid(n_tiles, G, n_splits);
  float* ws = n_splits > 1 ? workspace : nullptr;
  return mixer_by_dtype(dtype, "b200_biased_prompt_attn", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if constexpr (std::is_same_v<T, float>) {
      return fail(B200_ESHAPE, "b200_biased_prompt_attn: 16-bit dtypes only");
    } else {
      auto launch = [&](auto kern) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        kern<<<grid, 128, smem, static_cast<cudaStream_t>(stream)>>>(
            static_cast<T*>(out), static_cast<const T*>(q), q_stride, static_cast<const T*>(gate), gate_stride,
            static_cast<const T*>(k_pool), static_cast<const T*>(v_pool), block_tables, table_stride,
            reinterpret_cast<const AttnTile*>(tiles), tok_pos, bias_lut, lut_len, lut_in_smem, q_vec, scale, temp_coef,
            temp_every, H, G, dk, dv, block_size, ws, max_tile_tokens);
      };
      // decoded tokens over pages of whole 16-token tiles: b200_decode_rows.cu, where both sides' times stand; its two tensor maps cost the
      // host about 2 us, which shows where few tokens leave the step to the host (75 -> 77 us): one kernel all the same, so that a token's
      // result does not depend on the others
      const bool rows = ksplit && decode_rows(DecodeRows{out, q, q_stride, gate, gate_stride, k_pool, v_pool, block_tables, table_stride, tiles,
                                                         tok_pos, bias_lut, lut_len, scale, temp_coef, temp_every, H, G, block_size, ws,
                                                         max_tile_tokens, kSplitKeys},
                                              dk, dv, max_tile_tokens, n_tiles, n_splits, dtype, static_cast<cudaStream_t>(stream)) == 0;
      if (rows) {
      } else if (ksplit) {
        if (dv8 == 4) launch(biased_prompt_attn_mma_kernel<T, 4, true>);
        else if (dv8 == 8) launch(biased_prompt_attn_mma_kernel<T, 8, true>);
        else launch(biased_prompt_attn_mma_kernel<T, 16, true>);
      } else {
        if (dv8 == 4) launch(biased_prompt_attn_mma_kernel<T, 4, false>);
        else if (dv8 == 8) launch(biased_prompt_attn_mma_kernel<T, 8, false>);
        else launch(biased_prompt_attn_mma_kernel<T, 16, false>);
      }
      const int rc = check_launch("b200_biased_prompt_attn");
      if (rc != 0 || !ws) return rc;
      // launched while the CTAs above run; it waits for them on the device
      cudaLaunchAttribute early{};
      early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
      early.val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(n_tiles, max_tile_tokens, H);
      cfg.blockDim = dim3(128);
      cfg.stream = static_cast<cudaStream_t>(stream);
      cfg.attrs = &early;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, biased_split_merge_kernel<T>, static_cast<T*>(out), static_cast<const float*>(ws), static_cast<const T*>(gate),
                         gate_stride, reinterpret_cast<const AttnTile*>(tiles), tok_pos, H, dv);
      return check_launch("b200_biased_prompt_attn (merge)");
    }
  });
}

int b200_grouped_linear_supported(int K, int dtype) {
  return (dtype == B200_DTYPE_BF16 || dtype == B200_DTYPE_F16) && K > 0 && K % 8 == 0;
}

int b200_grouped_linear(void* out, const void* xs, const void* w, const int32_t* offsets, int64_t max_rows, int E, int N,
                        int K, int dtype, void* stream) {
  if (max_rows < 0 || E <= 0 || N <= 0 || K <= 0) return fail(B200_EINVAL, "b200_grouped_linear: bad sizes");
  if (!b200_grouped_linear_supported(K, dtype))
    return fail(B200_ESHAPE, "b200_grouped_linear: needs a 16-bit dtype and K %% 8 == 0");
  if (max_rows == 0) return 0;
  if (!out || !xs || !w || !offsets) return fail(B200_EINVAL, "b200_grouped_linear: null pointer");
  if (!aligned16(xs) || !aligned16(w)) return fail(B200_ESHAPE, "b200_grouped_linear: operands must be 16-byte aligned");
  const int64_t zt = (max_rows + kGrpRows - 1) / kGrpRows;
  if (zt > 65535 || E > 65535) return fail(B200_ENOSPC, "b200_grouped_linear: %lld row tiles / %d experts beyond the grid", static_cast<long long>(zt), E);
  const size_t smem = 2u * 2u * (kGrpRows + kGrpCols) * (kGrpK + 8);
  const dim3 grid((N + kGrpCols - 1) / kGrpCols, E, static_cast<unsigned>(zt));
  return mixer_by_dtype(dtype, "b200_grouped_linear", [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if constexpr (std::is_same_v<T, float>) {
      return fail(B200_ESHAPE, "b200_grouped_linear: 16-bit dtypes only");
    } else {
      auto kern = grouped_linear_kernel<T>;
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
      kern<<<grid, 128, smem, static_cast<cudaStream_t>(stream)>>>(static_cast<T*>(out), static_cast<const T*>(xs),
                                                                  static_cast<const T*>(w), offsets, N, K);
      return check_launch("b200_grouped_linear");
    }
  });
}

int b200_gated_scan(float* o_raw, const void* zq, const void* zf, const void* v, int64_t in_stride, const void* f_bias,
                    const void* lower, float* state, const int32_t* seqs, int n_seqs, int max_count, int H, int dk, int dv,
                    int dtype, void* stream) {
  if (n_seqs < 0 || H <= 0 || dk <= 0 || dv <= 0) return fail(B200_EINVAL, "b200_gated_scan: bad sizes");
  if (n_seqs == 0) return 0;
  if (!o_raw || !zq || !zf || !v || !f_bias || !lower || !state || !seqs) return fail(B200_EINVAL, "b200_gated_scan: null pointer");
  (void)max_count;   // one kernel for portions of any length (b200_split_scan: in chunks)
  if (2 * dk + 32 > 1024) return fail(B200_ESHAPE, "b200_gated_scan: key size %d beyond 496", dk);
  return gated_column_scan(o_raw, ScanRows{zq, zf, v, in_stride}, f_bias, lower, state, seqs, ScanShape{n_seqs, H, H, dk, dv}, dtype,
                           static_cast<cudaStream_t>(stream));
}

int b200_sigmoid_topk(int32_t* ids, float* weights, const float* logits, int n_tok, int E, int top, void* stream) {
  if (n_tok < 0 || E <= 0 || top <= 0 || top > E) return fail(B200_EINVAL, "b200_sigmoid_topk: bad sizes");
  if (n_tok == 0) return 0;
  if (!ids || !weights || !logits) return fail(B200_EINVAL, "b200_sigmoid_topk: null pointer");
  sigmoid_topk_kernel<<<(n_tok + 3) / 4, 128, 0, static_cast<cudaStream_t>(stream)>>>(ids, weights, logits, n_tok, E, top);
  return check_launch("b200_sigmoid_topk");
}

}  // extern "C"
