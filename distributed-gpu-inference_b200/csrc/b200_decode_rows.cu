// Attention of decoded tokens with a bias per (distance, head), a query temperature and an output gate: 16-bit types, head sizes 64 and
// 128, pages of whole 16-token tiles, up to 16 query rows per sequence and kv head.
//
// What bounds it: the keys and values, read once (48 sequences of up to 3000 tokens over 4 kv heads of 128 + 128: 246 MB, 38 us).  The
// kernel before (b200_mixer_ops.cu, still there for other shapes) moved its tiles with a copy instruction, a table look-up and an address
// per 16 bytes, put one set of keys into fragments with 4-byte reads for 16 rows of which four were live, and took two block barriers per
// 64 keys: 1450 instructions per warp and 16 keys, 95 us at 47 % issue and 2.6 TB/s.  Here a warp has 16-key tiles of its own, fetched by
// the copy engine into its own ring of two (no block barrier before the merge); keys stand where the matrix instruction has 16 rows and
// the query rows where it has eight columns; the bias of the next tile is asked for before this one is waited for.  Three CTAs per
// SM keep 192 KB under way.  Same case: 49.9 us.
//
// Every wait is bounded: a copy that does not land within a second ends its warp's walk, the copies still under way are waited for (a
// second again) before the merge takes their place, and the CTA's rows come out as NaN.
#include <cuda.h>

#include <atomic>
#include <type_traits>

#include "b200_common.cuh"
#include "b200_decode_rows.cuh"
#include "b200_tma_common.cuh"

namespace b200 {
namespace {

using namespace tma;

// Stages per warp: two, with three CTAs per SM where 168 registers do (rows in one eight); three stages and two CTAs, as much under way,
// showed more of a CTA's start, 59.5 us against 49.9 in the case above.  Key ranges of 512 instead of 256: 49.7.
constexpr int kStages = 2;

// false after about a second
__device__ __forceinline__ bool landed(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
    if (clock64() - t0 > 2000000000ll) return false;
  }
}

template <int DK, int DV>
struct Ring {
  static constexpr int kK = kTok * DK * 2, kV = kTok * DV * 2, kStage = kK + kV, kBytes = kWarps * kStages * kStage;
  static constexpr int kSmem = kBytes + kWarps * kStages * 8 + 1024;
};

// NB: query rows in eights
template <typename T, int DK, int DV, int NB>
__global__ void __launch_bounds__(kWarps * 32, NB == 1 ? 3 : 2)
decode_rows_kernel(const DecodeRows A, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map) {
  using R = Ring<DK, DV>;
  constexpr int KS = DK / 16, MT = DV / 16, ROWS = 8 * NB;
  static_assert(kWarps * ROWS * (DV + 2) * 4 <= R::kBytes, "the merge aliases the rings");
  asm volatile("griddepcontrol.launch_dependents;");
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane >> 2, tq = lane & 3;
  const uint32_t ring = smem_u32(smem) + warp * kStages * R::kStage;
  const uint32_t bars = smem_u32(smem + R::kBytes) + warp * kStages * 8;
  const int tok0 = A.tiles[3 * blockIdx.x], count = A.tiles[3 * blockIdx.x + 1], seq = A.tiles[3 * blockIdx.x + 2];
  const int g = blockIdx.y, rep = A.H / A.G, n_rows = count * rep;
  const int pos0 = A.tok_pos[tok0], p_last = pos0 + count - 1;
  const bool split = A.ws != nullptr;
  const int key_from = split ? blockIdx.z * A.split_keys : 0;
  const int keys = (split ? min(p_last + 1, key_from + A.split_keys) : p_last + 1) - key_from;
  if (keys <= 0) return;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < kStages; ++s) mbar_init(bars + s * 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  const int n_tiles = (keys + kTok - 1) / kTok, n_mine = n_tiles > warp ? (n_tiles - warp + kWarps - 1) / kWarps : 0;
  const int per_page = A.block_size / kTok, first = key_from / kTok + warp;      // tiles of the sequence: first, first + 4, ...
  const int32_t* table = A.block_tables + static_cast<int64_t>(seq) * A.table_stride;
  // lane l: the pool row (in tiles) of this warp's tile base + l; behind the context's last key the table is not read (its stride says
  // nothing about its width: one row may serve all sequences with stride 0)
  int base = 0;
  auto look_up = [&] {
    const int t = first + (base + lane) * kWarps;
    return t * kTok <= p_last ? (table[t / per_page] * A.G + g) * per_page + t % per_page : 0;
  };
  int rows16 = look_up();
  auto fetch = [&](int j) {
    if (j - base >= 32) {
      base += 32;
      rows16 = look_up();
    }
    const int row = __shfl_sync(0xffffffffu, rows16, j - base) * kTok;
    if (lane == 0) {
      const uint32_t bar = bars + j % kStages * 8, dst = ring + j % kStages * R::kStage;
      mbar_expect_tx(bar, R::kStage);
#pragma unroll
      for (int b = 0; b < DK / 64; ++b) tma_load_2d(dst + b * (kTok * 128), &k_map, b * 64, row, bar);
#pragma unroll
      for (int b = 0; b < DV / 64; ++b) tma_load_2d(dst + R::kK + b * (kTok * 128), &v_map, b * 64, row, bar);
    }
  };
  for (int j = 0; j < min(kStages, n_mine); ++j) fetch(j);

  // query row r = (token r / rep, head g rep + r % rep); this lane's columns are rows 8 b + 2 tq + c, its fragments row 8 b + quad
  uint32_t qf[NB][KS][2];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int r = 8 * b + quad, t = r / rep;
    const T* row = static_cast<const T*>(A.q) + (tok0 + t) * A.q_stride + (g * rep + r - t * rep) * DK + 2 * tq;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      qf[b][k][0] = r < n_rows ? *reinterpret_cast<const uint32_t*>(row + 16 * k) : 0u;
      qf[b][k][1] = r < n_rows ? *reinterpret_cast<const uint32_t*>(row + 16 * k + 8) : 0u;
    }
  }
  int pos[NB][2];
  const float* lut[NB][2];
  float qmul[NB][2], m[NB][2], l[NB][2], o[NB][MT][4], bias[NB][4];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int r = 8 * b + 2 * tq + c, t = r / rep;
      pos[b][c] = r < n_rows ? pos0 + t : -1;
      lut[b][c] = A.bias_lut + static_cast<int64_t>(g * rep + r - t * rep) * A.lut_len;
      qmul[b][c] = A.scale * (1.0f + A.temp_coef * logf(static_cast<float>((pos[b][c] + 1) / max(A.temp_every, 1)) + 1.0f));
      m[b][c] = -INFINITY;
      l[b][c] = 0.f;
    }
#pragma unroll
    for (int n = 0; n < MT; ++n) o[b][n][0] = o[b][n][1] = o[b][n][2] = o[b][n][3] = 0.f;
  }
  // element e of a score fragment: key quad + 8 (e >> 1) of the tile, column e & 1
  auto biases = [&](int i) {
    const int key = (first + i * kWarps) * kTok + quad;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = pos[b][e & 1] - key - 8 * (e >> 1);
        bias[b][e] = i < n_mine && d >= 0 ? lut[b][e & 1][min(d, A.lut_len - 1)] : 0.f;
      }
    }
  };
  biases(0);
  const int mat = lane >> 3, mrow = lane & 7;
  const int k_row = (mat & 1) * 8 + mrow, k_chunk = mat >> 1, v_row = (mat >> 1) * 8 + mrow, v_chunk = mat & 1;
  bool lost = false;
  for (int i = 0; i < n_mine; ++i) {
    const uint32_t kt = ring + i % kStages * R::kStage, vt = kt + R::kK;
    if (!__all_sync(0xffffffffu, landed(bars + i % kStages * 8, (i / kStages) & 1))) {
      for (int j = i; j < min(i + kStages, n_mine); ++j) landed(bars + j % kStages * 8, (j / kStages) & 1);
      lost = true;
      break;
    }
    const int key0 = (first + i * kWarps) * kTok;
    if (key0 + kTok > p_last + 1) zero_v_tail<DV>(vt, p_last + 1 - key0, lane);      // rows that nobody wrote
    float s[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b) s[b][0] = s[b][1] = s[b][2] = s[b][3] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      uint32_t a[4];
      ldmatrix_x4(a, kt + tile_off(k_row, 2 * k + k_chunk));
#pragma unroll
      for (int b = 0; b < NB; ++b) Mma<T>::run(s[b], a, qf[b][k][0], qf[b][k][1]);
    }
    uint32_t p[NB][2];
    float corr[NB][2];
    bool rescale = false;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        s[b][e] = key0 + quad + 8 * (e >> 1) <= pos[b][e & 1] ? s[b][e] * qmul[b][e & 1] + bias[b][e] : -INFINITY;
    }
    biases(i + 1);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float mx = fmaxf(s[b][c], s[b][c + 2]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float m_new = fmaxf(m[b][c], mx), safe = m_new == -INFINITY ? 0.f : m_new;      // a row that sees no key yet
        rescale |= m_new != m[b][c];
        corr[b][c] = expf(m[b][c] - safe);
        m[b][c] = m_new;
        s[b][c] = expf(s[b][c] - safe);
        s[b][c + 2] = expf(s[b][c + 2] - safe);
        l[b][c] = l[b][c] * corr[b][c] + (s[b][c] + s[b][c + 2]);
      }
      p[b][0] = movmatrix_trans(Mma<T>::pack(s[b][0], s[b][1]));
      p[b][1] = movmatrix_trans(Mma<T>::pack(s[b][2], s[b][3]));
    }
    if (__any_sync(0xffffffffu, rescale)) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
#pragma unroll
        for (int n = 0; n < MT; ++n) {
#pragma unroll
          for (int e = 0; e < 4; ++e) o[b][n][e] *= corr[b][e & 1];
        }
      }
    }
#pragma unroll
    for (int n = 0; n < MT; ++n) {
      uint32_t a[4];
      ldmatrix_x4_trans(a, vt + tile_off(v_row, 2 * n + v_chunk));
#pragma unroll
      for (int b = 0; b < NB; ++b) Mma<T>::run(o[b][n], a, p[b][0], p[b][1]);
    }
    __syncwarp();      // every lane has read the stage
    if (i + kStages < n_mine) fetch(i + kStages);
  }
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int w = 4; w < 32; w *= 2) l[b][c] += __shfl_xor_sync(0xffffffffu, l[b][c], w);
    }
  }
  // the warps' (maximum, sum, output) over the rings, taken together in their order
  const bool failed = __syncthreads_or(lost);
  float* o_s = reinterpret_cast<float*>(smem);      // [4][ROWS][DV]
  float* m_s = o_s + kWarps * ROWS * DV;
  float* l_s = m_s + kWarps * ROWS;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int n = 0; n < MT; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) o_s[(warp * ROWS + 8 * b + 2 * tq + (e & 1)) * DV + 16 * n + quad + 8 * (e >> 1)] = o[b][n][e];
    }
    if (quad == 0) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        m_s[warp * ROWS + 8 * b + 2 * tq + c] = m[b][c];
        l_s[warp * ROWS + 8 * b + 2 * tq + c] = l[b][c];
      }
    }
  }
  __syncthreads();
  const int64_t ws_row = (static_cast<int64_t>(blockIdx.z) * gridDim.x + blockIdx.x) * A.ws_tile;
  for (int i = threadIdx.x; i < n_rows * DV; i += kWarps * 32) {
    const int r = i / DV, c = i % DV, t = r / rep, h = g * rep + r - t * rep;
    float M = -INFINITY, L = 0.f, O = failed ? NAN : 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, m_s[w * ROWS + r]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = m_s[w * ROWS + r] == -INFINITY ? 0.f : expf(m_s[w * ROWS + r] - M);
      L = fmaf(l_s[w * ROWS + r], f, L);
      O = fmaf(o_s[(w * ROWS + r) * DV + c], f, O);
    }
    if (split) {
      float* dst = A.ws + ((ws_row + t) * A.H + h) * (DV + 2);
      dst[2 + c] = O;
      if (c == 0) {
        dst[0] = M;
        dst[1] = L;
      }
    } else {
      const int64_t n = tok0 + t;
      const float z = A.gate ? Cvt<T>::to_f32(static_cast<const T*>(A.gate)[n * A.gate_stride + h]) : 0.f;
      const float inv = (A.gate ? 1.0f / (1.0f + expf(-z)) : 1.0f) / L;
      static_cast<T*>(A.out)[(n * A.H + h) * DV + c] = Cvt<T>::from_f32(O * inv);
    }
  }
}

// The pool as rows of `width` elements in boxes of 64 columns x one tile; made for the launch (a microsecond) and not kept.
template <typename T>
bool tile_map(CUtensorMap* map, const void* pool, int width) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<Encode>(p);
  }();
  if (!encode) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(width), 0x7fffffffu}, strides[1] = {2ull * width};
  const cuuint32_t box[2] = {64, kTok}, step[2] = {1, 1};
  return encode(map, std::is_same_v<T, __nv_bfloat16> ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(pool),
                dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T, int DK, int DV>
int launch(const DecodeRows& A, int rows, dim3 grid, cudaStream_t stream) {
  CUtensorMap k_map, v_map;
  if (!tile_map<T>(&k_map, A.k_pool, DK) || !tile_map<T>(&v_map, A.v_pool, DV)) return 1;
  auto go = [&](auto nb) {      // a body, and so a flag, per kernel
    constexpr int smem = Ring<DK, DV>::kSmem;
    const auto kern = decode_rows_kernel<T, DK, DV, decltype(nb)::value>;
    static std::atomic<uint64_t> ready{0};      // a bit per device: the limit is always the same, a call need not set it again
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 64 || !(ready.load(std::memory_order_acquire) >> device & 1)) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (device < 64) ready.fetch_or(1ull << device, std::memory_order_release);
    }
    kern<<<grid, kWarps * 32, smem, stream>>>(A, k_map, v_map);
  };
  if (rows <= 8) go(std::integral_constant<int, 1>{});
  else go(std::integral_constant<int, 2>{});
  return 0;
}

}  // namespace

int decode_rows(const DecodeRows& A, int dk, int dv, int max_tile_tokens, int n_tiles, int n_splits, int dtype, cudaStream_t stream) {
  const int rows = max_tile_tokens * (A.H / A.G);
  if (rows <= 0 || rows > 16 || A.block_size % kTok || A.split_keys % kTok || A.G > 65535 || (dtype != B200_DTYPE_F16 && dtype != B200_DTYPE_BF16)) return 1;
  if (reinterpret_cast<uintptr_t>(A.q) % 4 || A.q_stride % 2 || !aligned16(A.k_pool) || !aligned16(A.v_pool)) return 1;
  const dim3 grid(n_tiles, A.G, n_splits);
  auto sized = [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    if (dk == 128 && dv == 128) return launch<T, 128, 128>(A, rows, grid, stream);
    if (dk == 64 && dv == 64) return launch<T, 64, 64>(A, rows, grid, stream);
    if (dk == 64 && dv == 128) return launch<T, 64, 128>(A, rows, grid, stream);
    if (dk == 128 && dv == 64) return launch<T, 128, 64>(A, rows, grid, stream);
    return 1;
  };
  return dtype == B200_DTYPE_F16 ? sized(static_cast<__half*>(nullptr)) : sized(static_cast<__nv_bfloat16*>(nullptr));
}

}  // namespace b200
