// Attention of prompt portions over the paged cache on the fifth-generation tensor cores (16-bit storage types).
//
// A CTA serves 128 query rows of one sequence and one kv head: up to 128 / rep consecutive tokens x the rep = H / G query heads that
// read this kv head, so a key tile is fetched once for all of them.  Keys are walked in tiles of 64.
//
//   S = Q K^T   tcgen05.mma, 128 x 64, both operands in shared memory (128-byte swizzled lines), S in tensor memory, two of them
//   P           256 threads, two per row: 32 scores each -> scale, query temperature, distance bias or soft cap, mask, running
//               maximum, exp2 in fp32; rounded to the storage type into the tensor memory S was in
//   O += P V    tcgen05.mma with P from tensor memory; V lies in shared memory as the pool holds it (one line per key), read with the
//               transposed descriptor; O stays in tensor memory in fp32 for the whole walk
//
// O is scaled down only when a row's maximum has grown by more than 2^8 since the reference its weights use (the weights then reach
// 256 at most, far inside both storage types, and the quotient O / l does not change): reading and writing O for every tile would
// cost as many tensor-memory accesses as the scores.  While the threads work on tile i the tensor cores run P V of tile i - 1; two
// CTAs share an SM where shared memory allows it (head sizes up to 128), so the products of one run under the softmax of the other.
// Pages arrive by cp.async a tile ahead (any page size; rows past the sequence are zero-filled).  A latent cache (values = the first
// DV columns of the key rows) is fetched once and read through both descriptors.
//
// Steps that give fewer CTAs than the chip has room for divide the keys over several CTAs (gridDim.z), which leave (maximum, sum,
// output) per row for the merge kernel of the older path.
//
// Every wait is bounded: a barrier that does not complete within a second marks the launch as failed, the rest of the walk does not
// wait, tensor memory is freed and the rows come out as NaN.
#include <algorithm>
#include <type_traits>

#include "../../include/b200_mixers.h"
#include "b200_common.cuh"
#include "b200_tile_attn.cuh"

namespace b200 {
namespace {

constexpr int kRows = kTileRows, kKeys = 64, kNT = 256;
constexpr int kBlk = kKeys * 128;        // bytes of 64 keys x 64 columns
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr float kSlack = 8.0f;           // growth of a row's maximum (in powers of two) that O is not rescaled for

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fence_smem_to_mma() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ bool bar_done(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// false when the barrier did not complete within about a second (or an earlier wait of the CTA already failed)
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* dead) {
  bool ok = bar_done(bar, parity);
  const long long t0 = clock64();
  while (!ok) {
    ok = bar_done(bar, parity);
    if (!ok && (*dead || clock64() - t0 > 2000000000ll)) {
      *dead = 1;
      break;
    }
  }
  __syncwarp();
  return ok;
}

// operand in 128-byte lines, 16-byte pieces swizzled by the line's number in its group of eight; `stride` between groups of eight
// lines, `lead` between blocks of 64 columns (transposed reads only)
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t lead, uint32_t stride) {
  return static_cast<uint64_t>((addr >> 4) & 0x3FFF) | (static_cast<uint64_t>((lead >> 4) & 0x3FFF) << 16) |
         (static_cast<uint64_t>((stride >> 4) & 0x3FFF) << 32) | (1ull << 46) | (2ull << 61);
}
template <typename T>
__device__ __forceinline__ constexpr uint32_t instr(int n, bool b_transposed) {
  constexpr uint32_t type = std::is_same_v<T, __nv_bfloat16> ? 1u : 0u;
  return (1u << 4) | (type << 7) | (type << 10) | (b_transposed ? 1u << 16 : 0u) | (static_cast<uint32_t>(n / 8) << 17) |
         (static_cast<uint32_t>(kRows / 16) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a),
               "l"(b), "r"(idesc), "r"(add ? 1u : 0u)
               : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a),
               "l"(b), "r"(idesc), "r"(add ? 1u : 0u)
               : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tm_ld32(float (&r)[32], uint32_t addr) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]),
        "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]),
        "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]),
        "=r"(u[30]), "=r"(u[31])
      : "r"(addr));
}
__device__ __forceinline__ void tm_st32(uint32_t addr, const float (&r)[32]) {
  const uint32_t* u = reinterpret_cast<const uint32_t*>(r);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),
      "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]),
      "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]), "r"(u[18]), "r"(u[19]), "r"(u[20]), "r"(u[21]), "r"(u[22]),
      "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]), "r"(u[27]), "r"(u[28]), "r"(u[29]), "r"(u[30]), "r"(u[31])
      : "memory");
}
__device__ __forceinline__ void tm_st16(uint32_t addr, const uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "r"(u[0]),
      "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]),
      "r"(u[13]), "r"(u[14]), "r"(u[15])
      : "memory");
}

__device__ __forceinline__ float exp2_fast(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (std::is_same_v<T, __nv_bfloat16>) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// shared memory of one CTA, from a 1024-byte boundary
template <int DK, int DV, bool ALIAS>
struct Plan {
  static constexpr int kKBufs = ALIAS ? 3 : 2;
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + DK / 64 * kRows * 128;
  static constexpr int kV = kK + kKBufs * (DK / 64) * kBlk;
  static constexpr int kEnd = kV + (ALIAS ? 0 : 2 * (DV / 64) * kBlk);
  static constexpr int kMax = kEnd;                    // float [2][2][128]: row maxima of the two halves, by tile parity
  static constexpr int kBar = kMax + 2 * 2 * kRows * 4;  // two barriers, the tensor memory's address, the failure flag
  static constexpr int kLut = kBar + 64;               // float [3][rep][pitch]: biases of the tiles' distances
  static constexpr int kO = 2 * kKeys;                 // columns of tensor memory: S0 | S1 | O
  static constexpr int kTm = kO + DV <= 256 ? 256 : 512;
};

template <typename T, int DK, int DV, bool ALIAS, bool BIAS>
__global__ void __launch_bounds__(kNT, DK <= 128 ? 2 : 1)
tile_attn_kernel(const TileAttn A) {
  using P = Plan<DK, DV, ALIAS>;
  extern __shared__ unsigned char raw_smem[];
  unsigned char* sm = raw_smem + ((1024 - (smem_u32(raw_smem) & 1023)) & 1023);
  const uint32_t sm0 = smem_u32(sm);
  float* mx_s = reinterpret_cast<float*>(sm + P::kMax);
  const uint32_t bar_s = sm0 + P::kBar, bar_o = bar_s + 8;
  volatile uint32_t* tm_slot = reinterpret_cast<volatile uint32_t*>(sm + P::kBar + 16);
  volatile int* dead = reinterpret_cast<volatile int*>(sm + P::kBar + 20);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = 32 * (warp & 3) + lane, half = warp >> 2;
  const int g = blockIdx.y, rep = A.H / A.G, bs = A.block_size;
  const int tok0 = A.tiles[3 * blockIdx.x], trow = A.tiles[3 * blockIdx.x + 2];
  const int cnt = min(A.tiles[3 * blockIdx.x + 1], kRows / rep), n_rows = cnt * rep;
  const int p0 = A.tok_pos[tok0], p_last = p0 + cnt - 1;
  const int32_t* table = A.block_tables + static_cast<int64_t>(trow) * A.table_stride;
  const T* kp = static_cast<const T*>(A.k_pool);
  const T* vp = static_cast<const T*>(A.v_pool);
  const int Gv = A.G / A.v_div, gv = g / A.v_div;
  const int bs_shift = (bs & (bs - 1)) == 0 ? __ffs(bs) - 1 : -1;
  auto first_seen = [&](int p) {
    int lo = A.window > 0 ? max(0, p - A.window + 1) : 0;
    if (A.chunk > 0) lo = max(lo, (p / A.chunk) * A.chunk);
    return lo;
  };
  // key tiles: those of the kept first tokens, then those from the first key the first token sees; this CTA's share of them
  const int lo0 = first_seen(p0);
  const int kf = A.window > 0 ? min(A.keep_first, lo0) : 0;
  const int nA = (kf + kKeys - 1) / kKeys;
  const int cB0 = max(nA, lo0 / kKeys), cB1 = p_last / kKeys;
  const int n_all = nA + cB1 - cB0 + 1;
  const int per = (n_all + gridDim.z - 1) / gridDim.z;
  const int it0 = blockIdx.z * per, n_it = min(n_all, it0 + per) - it0;
  auto key0 = [&](int i) {
    const int it = it0 + i;
    return (it < nA ? it : cB0 + it - nA) * kKeys;
  };

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_s));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_o));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *dead = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm0 + P::kBar + 16), "n"(P::kTm) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // ---- loads --------------------------------------------------------------------------------------------------------------
  auto page_row = [&](int j, int heads, int head) -> int64_t {
    const int b = bs_shift >= 0 ? j >> bs_shift : j / bs;
    return (static_cast<int64_t>(table[b]) * heads + head) * bs + (j - b * bs);
  };
  auto line = [](uint32_t base, int r, int ch, int rows) {     // 16-byte piece ch of row r: blocks of 64 columns, swizzled lines
    return base + (ch >> 3) * (rows * 128) + r * 128 + (((ch & 7) ^ (r & 7)) << 4);
  };
  {
    constexpr int kCh = DK / 8;
    const T* qp = static_cast<const T*>(A.q);
    for (int c = tid; c < kRows * kCh; c += kNT) {
      const int r = c / kCh, ch = c - r * kCh;
      const int t = r / rep, hh = g * rep + r - t * rep;
      const bool ok = r < n_rows;
      cp16(line(sm0 + P::kQ, r, ch, kRows), ok ? qp + (tok0 + t) * A.q_tok_stride + hh * A.q_head_stride + ch * 8 : qp, ok);
    }
  }
  auto load_rows = [&](uint32_t base, const T* pool, int heads, int head, int width, auto cols, int j0) {
    constexpr int kCh = decltype(cols)::value / 8;
#pragma unroll
    for (int u = 0; u < kKeys * kCh / kNT; ++u) {
      const int c = tid + u * kNT, key = c / kCh, ch = c - key * kCh, j = j0 + key;
      const bool ok = j <= p_last;
      cp16(line(base, key, ch, kKeys), ok ? pool + page_row(j, heads, head) * width + ch * 8 : pool, ok);
    }
  };
  const int pitch = ((cnt + kKeys - 1 + 31) & ~31) + (rep >= 32 ? 1 : 32 / rep);
  float* lut_s = reinterpret_cast<float*>(sm + P::kLut);
  auto load_bias = [&](int i) {       // entry [hh][x]: the bias of distance p0 - key0 - 63 + x
    if constexpr (BIAS) {
      const int d0 = p0 - key0(i) - (kKeys - 1), span = cnt + kKeys - 1;
      const uint32_t dst = smem_u32(lut_s + (i % 3) * rep * pitch);
      for (int e = tid; e < rep * span; e += kNT) {
        const int hh = e / span, x = e - hh * span;
        cp4(dst + 4 * (hh * pitch + x), A.bias_lut + static_cast<int64_t>(g * rep + hh) * A.lut_len + min(max(d0 + x, 0), A.lut_len - 1));
      }
    }
  };
  auto load_k = [&](int i) {
    if (i < n_it) {
      load_rows(sm0 + P::kK + (i % P::kKBufs) * (DK / 64) * kBlk, kp, A.G, g, DK, std::integral_constant<int, DK>{}, key0(i));
      if constexpr (BIAS) load_bias(i);
    }
    cp_commit();
  };
  auto load_v = [&](int i) {
    if constexpr (!ALIAS) {
      if (i < n_it) load_rows(sm0 + P::kV + (i & 1) * (DV / 64) * kBlk, vp, Gv, gv, A.v_row, std::integral_constant<int, DV>{}, key0(i));
      cp_commit();
    }
  };

  // ---- products, issued by one thread ---------------------------------------------------------------------------------------
  auto issue_scores = [&](int i, uint32_t tm) {
    const uint32_t k = sm0 + P::kK + (i % P::kKBufs) * (DK / 64) * kBlk;
#pragma unroll
    for (int kk = 0; kk < DK / 16; ++kk)
      mma_ss(tm + (i & 1) * kKeys, operand(sm0 + P::kQ + (kk >> 2) * (kRows * 128) + (kk & 3) * 32, 16, 1024),
             operand(k + (kk >> 2) * kBlk + (kk & 3) * 32, 16, 1024), instr<T>(kKeys, false), kk > 0);
    mma_commit(bar_s);
  };
  auto issue_values = [&](int i, uint32_t tm) {
    const uint32_t v = ALIAS ? sm0 + P::kK + (i % P::kKBufs) * (DK / 64) * kBlk : sm0 + P::kV + (i & 1) * (DV / 64) * kBlk;
#pragma unroll
    for (int kk = 0; kk < kKeys / 16; ++kk)
      mma_ts(tm + P::kO, tm + (i & 1) * kKeys + 8 * kk, operand(v + kk * 2048, kBlk, 1024), instr<T>(DV, true), i > 0 || kk > 0);
    mma_commit(bar_o);
  };

  // this thread's row
  const int t_row = row / rep, h_row = g * rep + row - t_row * rep;
  const bool live = row < n_rows;
  const int p = live ? p0 + t_row : -1;
  const int lo_p = live ? first_seen(p) : 0;
  float mult = A.scale;
  if (BIAS) mult *= 1.0f + A.temp_coef * logf(static_cast<float>((p + 1) / max(A.temp_every, 1)) + 1.0f);
  const float c2 = mult * kLog2e, two_over_cap = A.softcap > 0.f ? 2.0f / A.softcap : 0.f;
  float m_ref = -INFINITY, l = 0.f;

  load_k(0);
  load_k(1);
  load_v(0);
  cp_wait<ALIAS ? 1 : 2>();          // the queries and the first keys
  fence_smem_to_mma();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tm_slot;
  const uint32_t tm_row = tm + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
  bool ok = true;
  if (n_it > 0 && tid == 0) issue_scores(0, tm);
  __syncwarp();

  for (int i = 0; i < n_it; ++i) {
    ok = bar_wait(bar_s, i & 1, dead) && ok;
    tc_fence_after();
    if constexpr (!ALIAS) load_k(i + 2);        // the product that just completed was the last reader of that buffer
    const int j0 = key0(i);
    float s[32];
    tm_ld32(s, tm_row + (i & 1) * kKeys + half * 32);
    tc_wait_ld();
    // scores in powers of two
    if constexpr (BIAS) {
      const float* b = lut_s + (i % 3) * rep * pitch + (row - t_row * rep) * pitch + t_row + (kKeys - 1) - half * 32;
#pragma unroll
      for (int c = 0; c < 32; ++c) s[c] = fmaf(live ? b[-c] : 0.f, kLog2e, s[c] * c2);
    } else if (A.softcap > 0.f) {
#pragma unroll
      for (int c = 0; c < 32; ++c)
        s[c] = kLog2e * A.softcap * (1.0f - __fdividef(2.0f, __expf(s[c] * mult * two_over_cap) + 1.0f));
    } else {
#pragma unroll
      for (int c = 0; c < 32; ++c) s[c] *= c2;
    }
    // keys in sight of every token of the tile need no mask
    if (j0 + kKeys - 1 > p0 || j0 < first_seen(p_last) || cnt * rep < kRows) {
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const int j = j0 + half * 32 + c;
        if (!(j <= p && (j >= lo_p || (A.window > 0 && j < A.keep_first)))) s[c] = -INFINITY;
      }
    }
    float mx = s[0];
#pragma unroll
    for (int c = 1; c < 32; ++c) mx = fmaxf(mx, s[c]);
    float* ex = mx_s + (i & 1) * 2 * kRows;
    ex[half * kRows + row] = mx;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");    // the two warps of these 32 rows
    mx = fmaxf(mx, ex[(half ^ 1) * kRows + row]);
    if (i > 0) {
      ok = bar_wait(bar_o, (i - 1) & 1, dead) && ok;
      tc_fence_after();
      load_v(i + 1);
    } else {
      load_v(1);
    }
    if constexpr (ALIAS) load_k(i + 2);
    const bool grow = mx > m_ref + kSlack || (m_ref == -INFINITY && mx > -INFINITY);
    if (__any_sync(0xffffffffu, grow)) {
      const float corr = grow ? exp2_fast(m_ref - mx) : 1.0f;      // 0 where nothing was seen before
      if (grow) m_ref = mx;
      l *= corr;
      if (i > 0) {
#pragma unroll 1
        for (int c = 0; c < DV / 2; c += 32) {
          float o[32];
          tm_ld32(o, tm_row + P::kO + half * (DV / 2) + c);
          tc_wait_ld();
#pragma unroll
          for (int x = 0; x < 32; ++x) o[x] *= corr;
          tm_st32(tm_row + P::kO + half * (DV / 2) + c, o);
        }
      }
    }
    const float m_safe = m_ref == -INFINITY ? 0.f : m_ref;          // a row that sees no key yet keeps weights 0
    uint32_t w[16];
    float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
    for (int c = 0; c < 32; c += 2) {
      const float a = exp2_fast(s[c] - m_safe), b = exp2_fast(s[c + 1] - m_safe);
      sum0 += a;
      sum1 += b;
      w[c >> 1] = pack2<T>(a, b);
    }
    l += sum0 + sum1;
    tm_st16(tm_row + (i & 1) * kKeys + half * 16, w);
    tc_wait_st();
    cp_wait<ALIAS ? 1 : 2>();        // the next keys and (own pool) this tile's values are in
    fence_smem_to_mma();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      if (i + 1 < n_it) issue_scores(i + 1, tm);
      issue_values(i, tm);
    }
    __syncwarp();
  }
  if (n_it > 0) {
    ok = bar_wait(bar_o, (n_it - 1) & 1, dead) && ok;
    tc_fence_after();
  }
  cp_wait<0>();

  // ---- the rows' sums, sink, gate, output --------------------------------------------------------------------------------------
  mx_s[half * kRows + row] = l;
  __syncthreads();
  l += mx_s[(half ^ 1) * kRows + row];
  ok = ok && !*dead;
  const float m_nat = m_ref * kLn2;
  const int64_t n = tok0 + t_row;
  if (gridDim.z > 1) {
    float* dst = A.ws + ((static_cast<int64_t>(blockIdx.z) * A.n_tok + n) * A.H + h_row) * (DV + 2);
    if (live && half == 0) {
      dst[0] = ok ? m_nat : NAN;
      dst[1] = l;
    }
#pragma unroll 1
    for (int c = 0; c < DV / 2; c += 32) {
      float o[32];
      __syncwarp();
      if (n_it > 0) {
        tm_ld32(o, tm_row + P::kO + half * (DV / 2) + c);
        tc_wait_ld();
      }
      if (live) {
#pragma unroll
        for (int x = 0; x < 32; x += 2)
          *reinterpret_cast<float2*>(dst + 2 + half * (DV / 2) + c + x) = n_it > 0 ? make_float2(o[x], o[x + 1]) : make_float2(0.f, 0.f);
      }
    }
  } else {
    float f = 1.0f / l;
    if (A.sink && live) {
      const float sk = A.sink[h_row], M = fmaxf(m_nat, sk);
      const float e = expf(m_nat - M);
      f = e / (l * e + expf(sk - M));
    }
    if (!ok) f = NAN;
    const T* gate = static_cast<const T*>(A.gate);
    if (gate && live && !A.gate_dim) f *= 1.0f / (1.0f + expf(-Cvt<T>::to_f32(gate[n * A.gate_stride + h_row])));
#pragma unroll 1
    for (int c = 0; c < DV / 2; c += 32) {
      float o[32];
      __syncwarp();
      tm_ld32(o, tm_row + P::kO + half * (DV / 2) + c);
      tc_wait_ld();
      if (!live) continue;       // reconverges at the loop's head
      const int col = half * (DV / 2) + c;
#pragma unroll
      for (int x = 0; x < 32; ++x) {
        o[x] *= f;
        if (gate && A.gate_dim) o[x] *= 1.0f / (1.0f + expf(-Cvt<T>::to_f32(gate[n * A.gate_stride + h_row * A.gate_dim + col + x])));
      }
      const int64_t at = n * A.out_tok_stride + h_row * A.out_head_stride + col;
      if (A.out_f32) {
        float* dst = static_cast<float*>(A.out) + at;
#pragma unroll
        for (int x = 0; x < 32; x += 2) *reinterpret_cast<float2*>(dst + x) = make_float2(o[x], o[x + 1]);
      } else {
        T* dst = static_cast<T*>(A.out) + at;
        if (A.out_vec) {
#pragma unroll
          for (int x = 0; x < 32; x += 8)
            *reinterpret_cast<uint4*>(dst + x) = make_uint4(pack2<T>(o[x], o[x + 1]), pack2<T>(o[x + 2], o[x + 3]),
                                                            pack2<T>(o[x + 4], o[x + 5]), pack2<T>(o[x + 6], o[x + 7]));
        } else {
#pragma unroll
          for (int x = 0; x < 32; x += 2) *reinterpret_cast<uint32_t*>(dst + x) = pack2<T>(o[x], o[x + 1]);
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "n"(P::kTm));
}

template <typename T, int DK, int DV, bool ALIAS, bool BIAS>
int launch_tiles(const TileAttn& A, int n_tiles, int n_splits, cudaStream_t stream) {
  using P = Plan<DK, DV, ALIAS>;
  const int rep = A.H / A.G;
  size_t smem = 1024 + P::kLut;
  if (BIAS) smem += sizeof(float) * 3 * rep * (((kRows / rep + kKeys - 1 + 31) & ~31) + (rep >= 32 ? 1 : 32 / rep));
  // tensor memory (512 columns per SM) has room for two CTAs of 256 columns: shared memory admits no third one
  smem = std::max<size_t>(smem, P::kTm == 256 ? 80 * 1024 : 120 * 1024);
  if (smem > 227 * 1024) return fail(B200_ESHAPE, "b200_tile_attn: %zu bytes of shared memory", smem);
  auto kern = tile_attn_kernel<T, DK, DV, ALIAS, BIAS>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  kern<<<dim3(n_tiles, A.G, n_splits), kNT, smem, stream>>>(A);
  return check_launch("b200_tile_attn");
}

template <typename T>
int launch_shape(const TileAttn& A, int dk, int dv, bool alias, int n_tiles, int n_splits, cudaStream_t stream) {
  if (A.bias_lut) {
    if (!alias && dk == 128 && dv == 128) return launch_tiles<T, 128, 128, false, true>(A, n_tiles, n_splits, stream);
    if (!alias && dk == 64 && dv == 64) return launch_tiles<T, 64, 64, false, true>(A, n_tiles, n_splits, stream);
  } else {
    if (!alias && dk == 128 && dv == 128) return launch_tiles<T, 128, 128, false, false>(A, n_tiles, n_splits, stream);
    if (!alias && dk == 64 && dv == 64) return launch_tiles<T, 64, 64, false, false>(A, n_tiles, n_splits, stream);
    if (alias && dk == 256 && dv == 256) return launch_tiles<T, 256, 256, true, false>(A, n_tiles, n_splits, stream);
    if (alias && dk == 320 && dv == 256) return launch_tiles<T, 320, 256, true, false>(A, n_tiles, n_splits, stream);
  }
  return fail(B200_ESHAPE, "b200_tile_attn: head sizes %d / %d are not built", dk, dv);
}

}  // namespace

bool tile_attn_supported(int H, int G, int dk, int dv, bool alias, bool bias, int dtype) {
  if (dtype != B200_DTYPE_BF16 && dtype != B200_DTYPE_F16) return false;
  if (H <= 0 || G <= 0 || H % G || H / G > (bias ? 16 : kRows)) return false;
  if (alias) return !bias && dv == 256 && (dk == 256 || dk == 320);
  return dk == dv && (dk == 64 || dk == 128);
}

int tile_attn_splits(int n_tiles, int key_tiles, int G, int dk) {
  const int64_t ctas = static_cast<int64_t>(n_tiles) * G, room = (dk <= 128 ? 2 : 1) * kNumSMs;
  if (ctas <= 0 || ctas * 2 > room) return 1;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>({16, room / ctas, key_tiles / 3})));
}

int tile_attn_launch(const TileAttn& A, int dk, int dv, bool alias, int n_tiles, int n_splits, int dtype, cudaStream_t stream) {
  return dtype == B200_DTYPE_BF16 ? launch_shape<__nv_bfloat16>(A, dk, dv, alias, n_tiles, n_splits, stream)
                                  : launch_shape<__half>(A, dk, dv, alias, n_tiles, n_splits, stream);
}

}  // namespace b200
