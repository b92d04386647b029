// Attention of prompt portions over the paged cache on the fifth-generation tensor cores (16-bit storage types).
//
// A CTA serves 128 or 256 query rows of one sequence and one kv head: up to rows / rep consecutive tokens x the rep = H / G query heads that
// read this kv head, so a key tile is fetched once for all of them.  Keys are walked in tiles of 64.
//
//   S = Q K^T   tcgen05.mma, 128 x 64 per half of the rows, both operands in shared memory (128-byte swizzled lines), S in tensor
//               memory, two of them per half
//   P           four warps per half, one thread per row: scale, query temperature, distance bias or soft cap, mask, running maximum, exp2 in
//               fp32; rounded to the storage type into the tensor memory S was in
//   O += P V    tcgen05.mma with P from tensor memory; V lies in shared memory as the pool holds it (one line per key), read with the
//               transposed descriptor; O stays in tensor memory in fp32 for the whole walk
//
// Four more warps copy pages a tile or two ahead - pages that divide 64 keys by the copy engine, one box of 64 columns per page and block of
// columns, a sequence's last tile and other page sizes row by row with rows past the sequence zero-filled - another one issues the products,
// and four (where one CTA has the SM to itself) rescale O between the products of two tiles; they meet at mbarriers only.  While the softmax works
// on tile i the tensor cores run S of tile i + 1 and P V of tile i - 1.  Of 256 rows, the two halves' warps take turns with the exponentials.
// Queries of full tiles come by the copy engine; rows leave through shared memory in 16-byte pieces side by side.
//
// What bounds it: the softmax's chain from S to P, 2000 to 2400 clocks per tile of 64 keys x 256 rows (bias and maximum 850, exponentials 950 beside the
// other half's; the tensor cores need 1280, the exponentials alone 1024), and 9000 clocks of a CTA's beginning and end (of 22000: a row of the output
// written by one thread took 5000, queries in 16-byte pieces 5000, code of modes that a launch does not use two to eight thousand in instruction
// misses).  Rescaling by the softmax itself: 2900 clocks per tile.  Issue slots are taken 45 % of the time: what is no maximum, exponential or load goes two at a time
// (without: a tenth more instructions, 3 % of the biased kernel's time).
// Measured on B200 (bf16, us, before these / now, the kernel by itself): 8 x 2048 tokens, 16 heads over 4 kv heads of 128, plain 211 / 189, window of 512
// 139 / 117, with distance biases, query temperature and gate 278 / 198, soft cap 319 / 238; 5 x 1024 with a cap under a window of 512 60 / 45; latent 320
// / 256, 4 portions of 700 .. 1500 tokens of 16 heads behind 700, window 512: 98 / 76; 364 shapes and kinds of scores 0.87 times on average.
// Portions smaller than a tile have walks of one or two key tiles, which wait for instructions: 16 heads with keys of their own, plain, 64 x 96 tokens
// 41 / 41, 128 x 40 54 / 55, 256 x 20 102 / 102 (44, 61 and 116 with a loop for each way pages come and a loop for each form of the output in
// the kernel, a division for a CTA's place, barriers of the rescaling warps where there are none, and rows of no token written to shared memory).
//
// Weights are taken relative to the row's running maximum, so that the largest is 1 and loses nothing when P is rounded to the storage
// type; O is scaled down whenever a row of the warp has a new maximum.  (Scaling only once the maximum has grown by 2^8 leaves the largest weight anywhere in 1 .. 256, rounded
// like any other while the sum is not: scores of standard deviation 4 and 10 over 2048 keys came out 0.0013 and 0.0011 from float64 before
// the output's own rounding, 0.0005 and 0.0003 this way.)  A latent cache (values = the first DV columns of the key rows) is fetched once
// and read through both descriptors.
//
// Steps that give fewer CTAs than the chip has room for divide the keys over several CTAs (gridDim.z), which leave (maximum, sum,
// output) per row for the merge kernel of the older path.
//
// Every wait is bounded: a barrier that does not complete within a second marks the launch as failed, the rest of the walk does not
// wait, tensor memory is freed and the rows come out as NaN.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "../../include/b200_mixers.h"
#include "b200_common.cuh"
#include "b200_tile_attn.cuh"

namespace b200 {
namespace {

constexpr int kRows = kTileRows, kKeys = 64;
constexpr int kLoad = 128;                // threads that copy pages; kRows more per half do the softmax, one warp issues products
constexpr int kBlk = kKeys * 128;        // bytes of 64 keys x 64 columns
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
  // no memory clobber: the rows of the next copies may be looked up in between (the group's commit and wait carry it)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0));
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
__device__ __forceinline__ bool bar_wait1(uint32_t bar, uint32_t parity, volatile int* dead) {
  if (bar_done(bar, parity)) return true;
  const long long t0 = clock64();
  while (!bar_done(bar, parity)) {
    if (*dead || clock64() - t0 > 2000000000ll) {
      *dead = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* dead) {   // by a whole warp
  const bool ok = bar_wait1(bar, parity, dead);
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
// Executed by a whole warp: one elected lane issues.  Operands that are the same in all lanes stay in uniform registers that way; a
// branch on the lane makes every operand of every product pass through a register move, which was most of the walk's time.
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile(
      "{\n.reg .pred p, q;\nelect.sync _|q, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u)
      : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile(
      "{\n.reg .pred p, q;\nelect.sync _|q, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar)
      : "memory");
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
__device__ __forceinline__ void tm_ld16(float (&r)[16], uint32_t addr) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]),
        "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(addr));
}
__device__ __forceinline__ void tm_st16(uint32_t addr, const uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "r"(u[0]),
      "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]),
      "r"(u[13]), "r"(u[14]), "r"(u[15])
      : "memory");
}

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 both(float x) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ f32x2 pair(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void apart(float& a, float& b, f32x2 v) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a warp's 32 rows of N columns times the lanes' factors, W columns at a time
template <int N, int W>
__device__ __forceinline__ void scale_rows(uint32_t addr, float k) {
  const f32x2 kk = both(k);
#pragma unroll 1
  for (int c = 0; c < N; c += W) {
    float o[W];
    if constexpr (W == 16) tm_ld16(o, addr + c);
    else tm_ld32(o, addr + c);
    tc_wait_ld();
#pragma unroll
    for (int x = 0; x < W; x += 16) {
      uint32_t w[16];
#pragma unroll
      for (int u = 0; u < 16; u += 2) {
        float lo, hi;
        apart(lo, hi, mul2(pair(o[x + u], o[x + u + 1]), kk));
        w[u] = __float_as_uint(lo), w[u + 1] = __float_as_uint(hi);
      }
      tm_st16(addr + c + x, w);
    }
  }
}

__device__ __forceinline__ float exp2_fast(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// (a, b) <- (a, b) * k + m
__device__ __forceinline__ void scale_shift(float& a, float& b, f32x2 k, f32x2 m) {
  asm("{\n.reg .b64 t;\nmov.b64 t, {%0, %1};\nfma.rn.f32x2 t, t, %2, %3;\nmov.b64 {%0, %1}, t;\n}\n" : "+f"(a), "+f"(b) : "l"(k), "l"(m));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
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

// Columns c .. c + 31 of a lane's row to its warp's rows in shared memory, as type O, 16-byte pieces swizzled by the row's number in its group
// of eight
template <typename T, int DV, typename O>
__device__ __forceinline__ void stage_rows(const float (&o)[32], uint32_t rows, int c) {
  constexpr int kPieces = DV * sizeof(O) / 16, kPer = 16 / sizeof(O);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int x = 0; x < 32; x += kPer) {
    uint32_t w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = sizeof(O) == 4 ? __float_as_uint(o[x + u]) : pack2<T>(o[(x + 2 * u) % 32], o[(x + 2 * u + 1) % 32]);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rows + lane * (kPieces * 16) + ((((c + x) / kPer) ^ (lane & 7)) << 4)), "r"(w[0]), "r"(w[1]),
                 "r"(w[2]), "r"(w[3]) : "memory");
  }
}
// ... and from there to memory, so that lanes side by side write pieces side by side; at0: where a lane's row begins
template <typename O, int DV>
__device__ __forceinline__ void staged_out(uint32_t rows, bool live, O* out, int64_t at0) {
  constexpr int kPieces = DV * sizeof(O) / 16, kPer = 16 / sizeof(O), kRowsAtOnce = 32 / kPieces > 0 ? 32 / kPieces : 1;
  const int lane = threadIdx.x & 31;
  __syncwarp();
  const unsigned seen = __ballot_sync(0xffffffffu, live);
#pragma unroll 4
  for (int u = 0; u < kPieces; ++u) {
    const int r = kPieces >= 32 ? u * 32 / kPieces : u * kRowsAtOnce + lane / kPieces, piece = kPieces >= 32 ? (u * 32 + lane) % kPieces : lane % kPieces;
    const int64_t to = __shfl_sync(0xffffffffu, at0, r);
    if (seen >> r & 1) {
      uint4 v;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(rows + r * (kPieces * 16) + ((piece ^ (r & 7)) << 4)) : "memory");
      *reinterpret_cast<uint4*>(out + to + piece * kPer) = v;
    }
  }
}
// A warp's rows of O out of tensor memory in the forms that most launches do not have: gates per channel, fp32, rows off 16 bytes (not staged).  A
// function of its own keeps their code out of the kernel, whose short walks wait for instructions.
template <typename T, int DV>
__device__ __noinline__ void rows_out_other(uint32_t tm_o, uint32_t rows, float f, const T* gates, bool live, bool staged, bool out_f32, void* out, int64_t at0) {
#pragma unroll 1
  for (int c = 0; c < DV; c += 32) {
    float o[32];
    __syncwarp();
    tm_ld32(o, tm_o + c);
    tc_wait_ld();
#pragma unroll
    for (int x = 0; x < 32; ++x) o[x] *= f;
    if (gates && live) {      // after the row's factor: a gated row is the ungated one times its gates, to the bit
#pragma unroll
      for (int x = 0; x < 32; ++x) o[x] *= 1.0f / (1.0f + expf(-Cvt<T>::to_f32(gates[c + x])));
    }
    if (out_f32) {
      if (staged) {
        stage_rows<T, DV, float>(o, rows, c);
      } else if (live) {
        float* dst = static_cast<float*>(out) + at0 + c;
#pragma unroll
        for (int x = 0; x < 32; x += 2) *reinterpret_cast<float2*>(dst + x) = make_float2(o[x], o[x + 1]);
      }
    } else if (staged) {
      stage_rows<T, DV, T>(o, rows, c);
    } else if (live) {
      T* dst = static_cast<T*>(out) + at0 + c;
#pragma unroll
      for (int x = 0; x < 32; x += 2) *reinterpret_cast<uint32_t*>(dst + x) = pack2<T>(o[x], o[x + 1]);
    }
  }
  if (staged && out_f32) staged_out<float, DV>(rows, live, static_cast<float*>(out), at0);
  else if (staged) staged_out<T, DV>(rows, live, static_cast<T*>(out), at0);
}

// shared memory of one CTA, from a 1024-byte boundary
template <int DK, int DV, bool ALIAS, int HALVES, int CTAS>
struct Plan {
  static constexpr int kHalves = HALVES;                // sets of 128 rows
  static constexpr int kCtas = CTAS;                    // per SM
  // One CTA per SM: warps of their own rescale O.  (Two have no registers for them: their softmax does it.)
  static constexpr int kScale = kCtas == 1 ? kRows : 0;
  static constexpr int kSoft = kHalves * kRows, kNT = kSoft + kLoad + 32 + kScale;
  // 17 warps: five on a scheduler leave 96 registers each; the softmax takes 32 more from the warps that copy and rescale (8 x 128 + 8 x 64 + 96 = 17 x 96)
  static constexpr bool kSplitRegs = kNT == 17 * 32;
  // ... which a launch has to have: with fewer the softmax would wait for good
  static constexpr bool enough(int regs) { return regs * kNT >= kSoft * 128 + (kLoad + kScale) * 64 + 32 * regs; }
  static constexpr int kBufs = kCtas == 2 ? 2 : 3;      // of keys, and of values
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + kHalves * (DK / 64) * kRows * 128;
  static constexpr int kV = kK + kBufs * (DK / 64) * kBlk;
  static constexpr int kEnd = kV + (ALIAS ? 0 : kBufs * (DV / 64) * kBlk);
  static constexpr int kBar = kEnd;                    // barriers, the tensor memory's address, the failure flag
  static constexpr int kFlags = kBar + 240, kPage = kBar + 256;   // int [2][2][64]: rows of the pools that a tile's keys / values are in (-1: none)
  static constexpr int kCorr = kPage + 2 * 2 * kKeys * 4;     // float [2][rows]: what O is multiplied by before a tile
  static constexpr int kLut = kCorr + (kScale ? 2 * kSoft * 4 : 0);  // float [kLuts][rep][pitch]: biases of the tiles' distances
  // A tile's biases are copied once S of the tile kBufs before it is done, hence P V of the one two before that, hence its softmax:
  // the last reader known to be through is tile i - kBufs - 2.
  static constexpr int kLuts = kBufs + 2;
  static constexpr int kO = 2 * kKeys;                 // columns of tensor memory per half: S0 | S1 | O
  static constexpr int kHalfTm = DK <= 128 ? 256 : 512;
  static constexpr int kTm = kHalves * kHalfTm;
  static_assert(kO + DV <= kHalfTm, "tensor memory");
  static_assert(kHalves * kRows * DV * 4 <= kEnd, "rows on their way out");
};

enum Mode { kPlain, kBiased, kCapped };      // scores: as they are, with distance biases and query temperatures, with a soft cap

template <typename T, int DK, int DV, bool ALIAS, int MODE, int HALVES, int CTAS>
__global__ void __launch_bounds__(Plan<DK, DV, ALIAS, HALVES, CTAS>::kNT, CTAS)
tile_attn_kernel(const TileAttn A, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                 const __grid_constant__ CUtensorMap q_map) {
  using P = Plan<DK, DV, ALIAS, HALVES, CTAS>;
  constexpr int NB = P::kBufs, kSoft = P::kSoft;
  constexpr bool BIAS = MODE == kBiased, CAP = MODE == kCapped;      // a mode's code is all that its kernel has: first passes wait for instructions
  extern __shared__ unsigned char raw_smem[];
  unsigned char* sm = raw_smem + ((1024 - (smem_u32(raw_smem) & 1023)) & 1023);
  const uint32_t sm0 = smem_u32(sm);
  // barriers: queries in; keys of a buffer in, and read; values of a buffer in; P V of a value buffer done; per half: S of a buffer
  // done, P of a buffer written, factors of O known, O rescaled.  All readers of one wait for a tile before the tile that completes it again can get that far.
  const uint32_t bar_q = sm0 + P::kBar, bar_k = bar_q + 8, bar_ke = bar_k + 24, bar_v = bar_ke + 24, bar_o = bar_v + 24,
                 bar_s = bar_o + 24, bar_p = bar_s + 32, bar_c = bar_p + 32, bar_r = bar_c + 32;
  volatile uint32_t* tm_slot = reinterpret_cast<volatile uint32_t*>(sm + P::kFlags);
  volatile int* dead = reinterpret_cast<volatile int*>(sm + P::kFlags + 4);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  // all kv heads of a tile, then the next tile's: with the tiles in order of their keys, the longest first, short ones fill the last round
  const int tile = A.tile0 + blockIdx.y, g = blockIdx.x, rep = A.H / A.G, bs = A.block_size;
  const int tok0 = A.tiles[3 * tile], trow = A.tiles[3 * tile + 2];
  const int cnt = min(A.tiles[3 * tile + 1], kSoft / rep), n_rows = cnt * rep;
  const int halves = P::kHalves == 2 && n_rows > kRows ? 2 : 1;       // in use
  const int p0 = A.tok_pos[tok0], p_last = p0 + cnt - 1;
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
  const int pitch = ((cnt + kKeys - 1 + 31) & ~31) + (rep >= 32 ? 1 : 32 / rep);
  float* lut_s = reinterpret_cast<float*>(sm + P::kLut);

  if (tid == 0) {
    auto init = [](uint32_t bar, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); };
    init(bar_q, kSoft);
    for (int b = 0; b < NB; ++b) {
      init(bar_k + 8 * b, ALIAS ? kLoad : kLoad / 2);
      init(bar_ke + 8 * b, 1);
      init(bar_v + 8 * b, kLoad / 2);
      init(bar_o + 8 * b, 1);
    }
    for (int b = 0; b < 4; ++b) {
      init(bar_s + 8 * b, 1);
      init(bar_p + 8 * b, kRows);
      if (P::kScale) {
        init(bar_c + 8 * b, kRows);
        init(bar_r + 8 * b, kRows);
      }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *dead = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sm0 + P::kFlags), "n"(P::kTm) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = __shfl_sync(0xffffffffu, *tm_slot, 0);

  auto line = [](uint32_t base, int r, int ch, int rows) {     // 16-byte piece ch of row r: blocks of 64 columns, swizzled lines
    return base + (ch >> 3) * (rows * 128) + r * 128 + (((ch & 7) ^ (r & 7)) << 4);
  };
  // P V of tile i is done, for all rows
  auto values_done = [&](int i) { return bar_wait(bar_o + 8 * (i % NB), (i / NB) & 1, dead); };

  if (warp >= kSoft / 32 && warp < (kSoft + kLoad) / 32) {
    if constexpr (P::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // ---- the warps that copy pages: half of them keys, half values; a latent cache: all of them its rows ------------------------
    const bool values = !ALIAS && warp >= kSoft / 32 + kLoad / 64;
    constexpr int kTeam = ALIAS ? kLoad : kLoad / 2;
    const int me = (tid - kSoft) % kTeam;
    const T* pool = static_cast<const T*>(values ? A.v_pool : A.k_pool);
    const int heads = values ? A.G / A.v_div : A.G, head = values ? g / A.v_div : g, width = values ? A.v_row : DK;
    const int32_t* table = A.block_tables + static_cast<int64_t>(trow) * A.table_stride;
    const int shift = (bs & (bs - 1)) == 0 ? __ffs(bs) - 1 : -1;
    int* rows_s = reinterpret_cast<int*>(sm + P::kPage) + (values ? 2 * kKeys : 0);
    // A tile whose keys all exist and whose pages divide it is fetched page by page by the copy engine (boxes of 64 columns that land as
    // `line` has them), the others (a sequence's last) row by row with zeros behind the last.
    const bool boxes = A.boxes != 0;
    const int n_pages = boxes ? kKeys / bs : 0;
    constexpr int kLoadWarps = kTeam / 32;
    const int my_page = (me & 31) * kLoadWarps + me / 32;        // the warps take turns with the pages: a copy costs its warp a hundred clocks
    auto whole = [&](int i) { return boxes && i < n_it && key0(i) + kKeys - 1 <= p_last; };
    // the page of one key of a tile (or the tile's page number `me`), looked up by the team's first threads a tile ahead of its copies
    auto look_up = [&](int i) {
      if (whole(i)) return my_page < n_pages ? table[key0(i) / bs + my_page] : -1;
      const int j = key0(i) + me;
      return me < kKeys && i < n_it && j <= p_last ? table[shift >= 0 ? j >> shift : j / bs] : -1;
    };
    auto biases = [&](int i) {      // entry [hh][x]: the bias of distance p0 - key0 - 63 + x
      const int d0 = p0 - key0(i) - (kKeys - 1), span = cnt + kKeys - 1;
      const uint32_t dst = smem_u32(lut_s + (i % P::kLuts) * rep * pitch);
      for (int x = me; x < span; x += kTeam) {
        const float* src = A.bias_lut + static_cast<int64_t>(g * rep) * A.lut_len + min(max(d0 + x, 0), A.lut_len - 1);
        for (int hh = 0; hh < rep; ++hh, src += A.lut_len) cp4(dst + 4 * (hh * pitch + x), src);
      }
    };
    auto copy_pages = [&](int i, int page) {
      if (my_page < n_pages) {
        constexpr int kBox = 128;       // bytes of a box's row
        const int cols = values ? DV / 64 : DK / 64;
        const uint32_t base = (values ? sm0 + P::kV + (i % NB) * (DV / 64) * kBlk : sm0 + P::kK + (i % NB) * (DK / 64) * kBlk) + my_page * bs * kBox;
        if (page >= 0) {
          const uint32_t bar = (values ? bar_v : bar_k) + 8 * (i % NB);
          asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(cols * bs * kBox) : "memory");
          for (int c = 0; c < cols; ++c)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(base + c * kBlk),
                         "l"(values ? &v_map : &k_map), "r"(64 * c), "r"((page * heads + head) * bs), "r"(bar) : "memory");
        } else {                        // no page: zeros
          for (int c = 0; c < cols; ++c) {
            for (int b = 0; b < bs * kBox; b += 16) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(base + c * kBlk + b), "r"(0) : "memory");
          }
        }
      }
      if (BIAS && !values) biases(i);
      cp_commit();
    };
    auto copy = [&](int i, int page) {
      if (whole(i)) return copy_pages(i, page);
      if (me < kKeys) {
        const int j = key0(i) + me, off = shift >= 0 ? j & (bs - 1) : j % bs;
        rows_s[(i & 1) * kKeys + me] = page < 0 ? -1 : (page * heads + head) * bs + off;
      }
      asm volatile("bar.sync %0, %1;" ::"r"(values ? 2 : 1), "n"(kTeam) : "memory");
      const uint32_t base = values ? sm0 + P::kV + (i % NB) * (DV / 64) * kBlk : sm0 + P::kK + (i % NB) * (DK / 64) * kBlk;
      auto move = [&](auto cols) {
        constexpr int kCh = decltype(cols)::value / 8;
        constexpr int kPer = kKeys * kCh / kTeam, kBatch = kPer % 8 == 0 ? 8 : (kPer % 10 == 0 ? 10 : 4);
        static_assert(kPer % kBatch == 0, "copies per thread");
#pragma unroll 1
        for (int u0 = 0; u0 < kPer; u0 += kBatch) {
          int r[kBatch];
#pragma unroll
          for (int u = 0; u < kBatch; ++u) r[u] = rows_s[(i & 1) * kKeys + (me + (u0 + u) * kTeam) / kCh];
#pragma unroll
          for (int u = 0; u < kBatch; ++u) {
            const int c = me + (u0 + u) * kTeam, key = c / kCh, ch = c - key * kCh;
            cp16(line(base, key, ch, kKeys), r[u] >= 0 ? pool + static_cast<int64_t>(r[u]) * width + ch * 8 : pool, r[u] >= 0);
          }
        }
      };
      if (DK == DV || !values) move(std::integral_constant<int, DK>{});
      else move(std::integral_constant<int, DV>{});
      if (BIAS && !values) biases(i);
      cp_commit();
    };
    auto arrived = [&](int i) {     // this thread's copies of the tile are in shared memory, for the tensor cores too
      fence_smem_to_mma();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((values ? bar_v : bar_k) + 8 * (i % NB)) : "memory");
    };
    int page = look_up(0);
    auto free_again = [&](int i) {      // the buffer that tile i goes into has been read
      if (values || ALIAS) values_done(i - NB);
      else bar_wait(bar_ke + 8 * (i % NB), (i / NB - 1) & 1, dead);
    };
    // Pages by the copy engine arrive at the barrier by themselves, biases by their own arrival: nobody waits for a tile before the next
    // is asked for.  Row by row a tile is handed over while the next one is under way, until the buffers are full.  One loop for both: the
    // copies' code is there once.
    for (int i = 0; i < n_it; ++i) {
      const int next = look_up(i + 1);
      if (i >= NB) free_again(i);
      copy(i, page);
      page = next;
      if (!boxes && i < NB) {
        if (i > 0) {
          cp_wait<1>();
          arrived(i - 1);
        }
        if (i + 1 < min(n_it, NB)) continue;
      }
      if (BIAS && !values && whole(i)) {
        fence_smem_to_mma();
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_k + 8 * (i % NB)) : "memory");
      } else {
        if (!whole(i)) cp_wait<0>();
        arrived(i);
      }
    }
  } else if (warp == (kSoft + kLoad + P::kScale) / 32) {
    // ---- products -----------------------------------------------------------------------------------------------------------------
    {
      auto scores = [&](int i) {
        const uint32_t k = sm0 + P::kK + (i % NB) * (DK / 64) * kBlk;
        bar_wait(bar_k + 8 * (i % NB), (i / NB) & 1, dead);
        tc_fence_after();
        for (int hf = 0; hf < halves; ++hf) {
#pragma unroll
          for (int kk = 0; kk < DK / 16; ++kk)
            mma_ss(tm + hf * P::kHalfTm + (i & 1) * kKeys,
                   operand(sm0 + P::kQ + (hf * (DK / 64) + (kk >> 2)) * (kRows * 128) + (kk & 3) * 32, 16, 1024),
                   operand(k + (kk >> 2) * kBlk + (kk & 3) * 32, 16, 1024), instr<T>(kKeys, false), kk > 0);
          mma_commit(bar_s + 16 * hf + 8 * (i & 1));
        }
        if (!ALIAS) mma_commit(bar_ke + 8 * (i % NB));
      };
      bar_wait(bar_q, 0, dead);
      if (n_it > 0) scores(0);
      for (int i = 0; i < n_it; ++i) {
        if (i + 1 < n_it) {
          // S of tile i + 1 goes where P of tile i - 1 is being read
          if (i > 0) bar_wait(bar_o + 8 * ((i - 1) % NB), ((i - 1) / NB) & 1, dead);
          scores(i + 1);
        }
        if (!ALIAS) bar_wait(bar_v + 8 * (i % NB), (i / NB) & 1, dead);
        const uint32_t v = ALIAS ? sm0 + P::kK + (i % NB) * (DK / 64) * kBlk : sm0 + P::kV + (i % NB) * (DV / 64) * kBlk;
        for (int hf = 0; hf < halves; ++hf) {
          bar_wait(bar_p + 16 * hf + 8 * (i & 1), (i >> 1) & 1, dead);
          if (P::kScale && i > 0) bar_wait(bar_r + 16 * hf + 8 * (i & 1), ((i - 1) >> 1) & 1, dead);
          tc_fence_after();
          const uint32_t t = tm + hf * P::kHalfTm;
#pragma unroll
          for (int kk = 0; kk < kKeys / 16; ++kk)
            mma_ts(t + P::kO, t + (i & 1) * kKeys + 8 * kk, operand(v + kk * 2048, kBlk, 1024), instr<T>(DV, true), i > 0 || kk > 0);
        }
        mma_commit(bar_o + 8 * (i % NB));
      }
    }
    __syncwarp();
  } else if (P::kScale && warp >= (kSoft + kLoad) / 32) {
    if constexpr (P::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // ---- O to a tile's new maximum, between P V of the tile before and the tile's own: not on the softmax's way from tile to tile ----
    const uint32_t quarter = static_cast<uint32_t>(32 * (warp & 3)) << 16;
    const float* corr_s = reinterpret_cast<const float*>(sm + P::kCorr) + 32 * (warp & 3) + (tid & 31);
    for (int i = 1; i < n_it; ++i) {
      for (int hf = 0; hf < halves; ++hf) {
        bar_wait(bar_c + 16 * hf + 8 * (i & 1), ((i - 1) >> 1) & 1, dead);
        const float corr = corr_s[(i & 1) * kSoft + hf * kRows];
        if (__any_sync(0xffffffffu, corr != 1.0f)) {
          values_done(i - 1);
          tc_fence_after();
          scale_rows<DV, 32>(tm + hf * P::kHalfTm + quarter + P::kO, corr);
          tc_wait_st();
          tc_fence_before();
        }
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_r + 16 * hf + 8 * (i & 1)) : "memory");
      }
    }
  } else {
    // ---- softmax: thread = row -------------------------------------------------------------------------------------------------------
    if constexpr (P::kSplitRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
    if (A.q_boxes && n_rows == kSoft) {
      // a full tile: boxes of 64 columns x the group's heads x the tokens of 128 rows
      if (tid == 0) {
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar_q), "n"(kSoft * DK * 2) : "memory");
        for (int c = 0; c < P::kHalves * (DK / 64); ++c)
          asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(sm0 + P::kQ + c * (kRows * 128)),
                       "l"(&q_map), "r"(64 * (c % (DK / 64))), "r"(g * rep), "r"(tok0 + c / (DK / 64) * (kRows / rep)), "r"(bar_q) : "memory");
      }
      __syncwarp();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_q) : "memory");
    } else {
      constexpr int kCh = DK / 8;
      const T* qp = static_cast<const T*>(A.q);
#pragma unroll 8
      for (int u = 0; u < kCh; ++u) {
        const int c = tid + u * kSoft, r = c / kCh, ch = c - r * kCh;
        const int t = r / rep, hh = g * rep + r - t * rep;
        const bool in = r < n_rows;
        cp16(line(sm0 + P::kQ + (r / kRows) * (DK / 64) * (kRows * 128), r % kRows, ch, kRows), in ? qp + (tok0 + t) * A.q_tok_stride + hh * A.q_head_stride + ch * 8 : qp, in);
      }
      cp_commit();
      cp_wait<0>();
      fence_smem_to_mma();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_q) : "memory");
    }
    const int hf = tid / kRows;
    const uint32_t tm_row = tm + hf * P::kHalfTm + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
    const uint32_t my_s = bar_s + 16 * hf, my_p = bar_p + 16 * hf;
    const int mine = hf < halves ? n_it : 0;
    const int row = tid, t_row = row / rep, hh = row - t_row * rep, h_row = g * rep + hh;
    const bool live = row < n_rows;
    const int p = live ? p0 + t_row : -1;
    const int lo_p = live ? first_seen(p) : 0, lo_last = first_seen(p_last);
    float mult = A.scale;
    if (BIAS) mult *= 1.0f + A.temp_coef * logf(static_cast<float>((p + 1) / max(A.temp_every, 1)) + 1.0f);
    [[maybe_unused]] const float two_over_cap = CAP ? 2.0f / A.softcap : 0.f;
    // plain scores are compared before they are scaled: weight = 2^(s * k2 - m), in one multiply-add
    const bool plain = MODE == kPlain && mult > 0.f;
    const float k2 = plain ? mult * kLog2e : kLog2e;
    float m_ref = -INFINITY, l = 0.f;       // in powers of two; -inf until the row sees a key
    bool ok = true;

    // O of the tiles before tile i to the new maximum where a row of the warp has one, with two CTAs per SM: before the tile's weights, as
    // their 96 registers do not hold the factor as well (after them 3 .. 12% slower)
    [[maybe_unused]] auto rescale = [&](int i, bool grow, float corr) {
      if (i == 0 || !__any_sync(0xffffffffu, grow)) return;
      ok = values_done(i - 1) && ok;
      tc_fence_after();
      scale_rows<DV, 16>(tm_row + P::kO, corr);
    };
    [[maybe_unused]] float* corr_s = reinterpret_cast<float*>(sm + P::kCorr);
    // Two warps share a scheduler, one of each half: they take turns with the exponentials, so that one's run under the other's maxima and
    // rescaling (in step, each phase is waited for twice)
    const bool turns = P::kHalves == 2 && halves == 2;
    const int turn_bar = 3 + 2 * (warp & 3);
    auto my_turn = [&](int i) {
      if (turns && (hf > 0 || i > 0)) asm volatile("bar.sync %0, 64;" ::"r"(turn_bar + hf) : "memory");
    };
    auto their_turn = [&](int i) {
      if (turns && (hf == 0 || i + 1 < mine)) asm volatile("bar.arrive %0, 64;" ::"r"(turn_bar + 1 - hf) : "memory");
    };
    for (int i = 0; i < mine; ++i) {
      const int j0 = key0(i);
      ok = bar_wait(my_s + 8 * (i & 1), (i >> 1) & 1, dead) && ok;
      tc_fence_after();
      float s[2][32];
      tm_ld32(s[0], tm_row + (i & 1) * kKeys);
      tm_ld32(s[1], tm_row + (i & 1) * kKeys + 32);
      tc_wait_ld();
      if constexpr (BIAS) {
        const float* b = lut_s + ((i % P::kLuts) * rep + (live ? hh : 0)) * pitch + (live ? t_row : 0) + kKeys - 1;
#pragma unroll
        for (int c = 0; c < kKeys; c += 2) {
          float& x = s[c >> 5][c & 31];
          float& y = s[c >> 5][(c & 31) + 1];
          apart(x, y, fma2(pair(x, y), both(mult), pair(b[-c], b[-c - 1])));
        }
      } else if (!plain) {
        [[maybe_unused]] float far = 0.f;
#pragma unroll
        for (int c = 0; c < kKeys; c += 2) {
          float& x = s[c >> 5][c & 31];
          float& y = s[c >> 5][(c & 31) + 1];
          apart(x, y, mul2(pair(x, y), both(mult)));
          if constexpr (CAP) far = max3(far, fabsf(x), fabsf(y));
        }
        if constexpr (!CAP) {
        } else if (!__any_sync(0xffffffffu, far > 0.5f * A.softcap)) {
          // all within half the cap: x tanh(u) / u, u = x / cap, by its series in u^2 (Chebyshev nodes on 0 .. 1/4, 3e-10): 1 / (1 + e^x) and
          // the difference from 1 took three times as long (5 x 1024 tokens of 16 heads, window 512: 99 us against 56) and lost the last
          // digits of small scores
          const f32x2 per_cap = both(0.5f * two_over_cap);
#pragma unroll
          for (int c = 0; c < kKeys; c += 2) {
            const f32x2 x = pair(s[c >> 5][c & 31], s[c >> 5][(c & 31) + 1]), u = mul2(x, per_cap), t = mul2(u, u);
            f32x2 q = fma2(t, both(-0x1.b12a58p-8f), both(0x1.5c8676p-6f));
            q = fma2(t, q, both(-0x1.b97d94p-5f));
            q = fma2(t, q, both(0x1.110ec8p-3f));
            q = fma2(t, q, both(-0x1.555550p-2f));
            apart(s[c >> 5][c & 31], s[c >> 5][(c & 31) + 1], fma2(mul2(x, t), q, x));
          }
        } else {
#pragma unroll
          for (int c = 0; c < kKeys; ++c) {
            float& x = s[c >> 5][c & 31];
            x = A.softcap * (1.0f - __fdividef(2.0f, __expf(x * two_over_cap) + 1.0f));
          }
        }
      }
      // keys in sight of every token of the tile need no mask
      if (j0 + kKeys - 1 > p0 || j0 < lo_last || n_rows < halves * kRows) {
#pragma unroll
        for (int c = 0; c < kKeys; ++c) {
          const int j = j0 + c;
          if (!(j <= p && (j >= lo_p || (A.window > 0 && j < A.keep_first)))) s[c >> 5][c & 31] = -INFINITY;
        }
      }
      float mx[4] = {s[0][0], s[0][1], s[0][2], s[0][3]};
#pragma unroll
      for (int c = 4; c < kKeys - 4; c += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u) mx[u] = max3(mx[u], s[c >> 5][(c & 31) + u], s[(c + 4) >> 5][((c + 4) & 31) + u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) mx[u] = fmaxf(mx[u], s[1][28 + u]);
      const float m_new = max3(mx[0], mx[1], fmaxf(mx[2], mx[3])) * k2;
      const bool grow = m_new > m_ref;
      const float corr = grow ? exp2_fast(m_ref - m_new) : 1.0f;      // 0 where nothing was seen before
      if (grow) m_ref = m_new;
      if constexpr (P::kScale > 0) {
        if (i > 0) {
          corr_s[(i & 1) * kSoft + tid] = corr;
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_c + 16 * hf + 8 * (i & 1)) : "memory");
        }
      } else {
        rescale(i, grow, corr);
      }
      const f32x2 kk = both(k2);
      f32x2 mm = both(m_ref == -INFINITY ? 0.f : -m_ref);     // a row that sees no key yet keeps weights 0
      f32x2 sum[2] = {0ull, 0ull};
      my_turn(i);
      asm volatile("" : "+l"(mm));        // no exponential before it
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t w[16];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float a = s[x][c], b = s[x][c + 1];
          scale_shift(a, b, kk, mm);
          a = exp2_fast(a);
          b = exp2_fast(b);
          sum[(c >> 1) & 1] = add2(sum[(c >> 1) & 1], pair(a, b));
          w[c >> 1] = pack2<T>(a, b);
        }
        tm_st16(tm_row + (i & 1) * kKeys + x * 16, w);
      }
      their_turn(i);
      float part[4];
      apart(part[0], part[1], sum[0]);
      apart(part[2], part[3], sum[1]);
      l = fmaf(l, corr, (part[0] + part[1]) + (part[2] + part[3]));
      tc_wait_st();
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(my_p + 8 * (i & 1)) : "memory");
    }
    if (mine > 0) {
      ok = values_done(n_it - 1) && ok;
      tc_fence_after();
    }

    // ---- sink, gate, output --------------------------------------------------------------------------------------------------------
    ok = ok && !*dead;
    const float m_nat = m_ref * kLn2;
    const int64_t n = tok0 + t_row;
    if (gridDim.z > 1) {
      const int64_t wr = (static_cast<int64_t>(blockIdx.z) * A.n_tiles + tile) * (kSoft / rep) + t_row;
      float* dst = A.ws + (wr * A.H + h_row) * (DV + 2);
      if (live) {
        dst[0] = ok ? m_nat : NAN;
        dst[1] = l;
      }
#pragma unroll 1
      for (int c = 0; c < DV; c += 32) {
        float o[32];
        __syncwarp();
        if (n_it > 0) {
          tm_ld32(o, tm_row + P::kO + c);
          tc_wait_ld();
        }
        if (live) {
#pragma unroll
          for (int x = 0; x < 32; x += 2)
            *reinterpret_cast<float2*>(dst + 2 + c + x) = n_it > 0 ? make_float2(o[x], o[x + 1]) : make_float2(0.f, 0.f);
        }
      }
    } else if (__any_sync(0xffffffffu, p >= 0)) {      // (p >= 0: live; the rows' number need not be kept)
      float f = 1.0f / l;
      if (A.sink && p >= 0) {
        const float sk = A.sink[h_row], M = fmaxf(m_nat, sk);
        const float e = expf(m_nat - M);
        f = e / (l * e + expf(sk - M));
      }
      if (!ok) f = NAN;
      const T* gate = static_cast<const T*>(A.gate);
      if (gate && p >= 0 && !A.gate_dim) f *= 1.0f / (1.0f + expf(-Cvt<T>::to_f32(gate[n * A.gate_stride + h_row])));
      const bool staged = A.out_vec && __all_sync(0xffffffffu, ok);     // after a failure copies may still be under way
      const int64_t at0 = n * A.out_tok_stride + h_row * A.out_head_stride;
      // the warp's own rows (all products are done, queries and pages have been read)
      const uint32_t own = sm0 + P::kQ + (hf * kRows + 32 * (warp & 3)) * (DV * 4);
      if (!staged || A.out_f32 || (gate && A.gate_dim)) {
        const T* gates = gate && A.gate_dim ? gate + n * A.gate_stride + h_row * A.gate_dim : nullptr;
        rows_out_other<T, DV>(tm_row + P::kO, own, f, gates, p >= 0, staged, A.out_f32 != 0, A.out, at0);
      } else {
#pragma unroll 1
        for (int c = 0; c < DV; c += 32) {
          float o[32];
          __syncwarp();
          tm_ld32(o, tm_row + P::kO + c);
          tc_wait_ld();
#pragma unroll
          for (int x = 0; x < 32; ++x) o[x] *= f;
          stage_rows<T, DV, T>(o, own, c);
        }
        staged_out<T, DV>(own, p >= 0, static_cast<T*>(A.out), at0);
      }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "n"(P::kTm));
}

using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                            const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
Encode tensor_map_encode() {
  static const Encode encode = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<Encode>(p);
  }();
  return encode;
}

// The pool as rows of `width` elements, fetched in boxes of 64 columns x one page; made for the launch (a microsecond) and not kept.
// Its height is the largest a row's number allows: which rows are read is the block tables' business, as with plain loads.
template <typename T>
bool page_map(CUtensorMap* map, const void* pool, int width, int block_size) {
  const Encode encode = tensor_map_encode();
  if (!encode || !aligned16(pool)) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(width), 0x7fffffffu}, strides[1] = {2ull * width};
  const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(block_size)}, step[2] = {1, 1};
  return encode(map, std::is_same_v<T, __nv_bfloat16> ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(pool),
                dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Queries as boxes of 64 columns x one kv head's heads x the tokens of 128 rows.  Only full tiles are fetched this way, so the number of
// tokens does not matter.
template <typename T>
bool query_map(CUtensorMap* map, const TileAttn& A, int dk) {
  const int rep = A.H / A.G;
  const Encode encode = tensor_map_encode();
  if (!encode || kRows % rep || A.q_head_stride <= 0 || A.q_tok_stride <= 0) return false;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(dk), static_cast<cuuint64_t>(A.H), 0x7fffffffu};
  const cuuint64_t strides[2] = {2ull * A.q_head_stride, 2ull * A.q_tok_stride};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(rep), static_cast<cuuint32_t>(kRows / rep)}, step[3] = {1, 1, 1};
  return encode(map, std::is_same_v<T, __nv_bfloat16> ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(A.q), dims,
                strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Registers per thread that a kernel was built with, which every device runs; a query that fails is not kept.
template <typename T, int DK, int DV, bool ALIAS, int MODE, int HALVES, int CTAS>
cudaError_t built_registers(int* regs) {
  static std::atomic<int> known{0};
  *regs = known.load(std::memory_order_relaxed);
  if (*regs > 0) return cudaSuccess;
  cudaFuncAttributes f{};
  const cudaError_t e = cudaFuncGetAttributes(&f, tile_attn_kernel<T, DK, DV, ALIAS, MODE, HALVES, CTAS>);
  if (e == cudaSuccess) known.store(*regs = f.numRegs, std::memory_order_relaxed);
  return e;
}
// Whether the kernels of 256 rows were built with the registers that they share out (unknown: yes, their launches ask again)
template <typename T, int D>
bool wide_built() {
  auto fits = [](auto mode) {
    int regs = 0;
    if (built_registers<T, D, D, false, decltype(mode)::value, 2, 1>(&regs) == cudaSuccess) return Plan<D, D, false, 2, 1>::enough(regs);
    cudaGetLastError();
    return true;
  };
  return fits(std::integral_constant<int, kPlain>{}) && fits(std::integral_constant<int, kBiased>{}) && fits(std::integral_constant<int, kCapped>{});
}

template <typename T, int DK, int DV, bool ALIAS, int MODE, int HALVES, int CTAS>
int launch_tiles(const TileAttn& A, int n_tiles, int n_splits, cudaStream_t stream) {
  using P = Plan<DK, DV, ALIAS, HALVES, CTAS>;
  const int rep = A.H / A.G;
  size_t smem = 1024 + P::kLut;
  if (MODE == kBiased) smem += sizeof(float) * P::kLuts * rep * (((P::kSoft / rep + kKeys - 1 + 31) & ~31) + (rep >= 32 ? 1 : 32 / rep));
  smem = std::max<size_t>(smem, P::kCtas == 2 ? 80 * 1024 : 120 * 1024);   // no more CTAs per SM than tensor memory has room for
  if (smem > kMaxSmem) return fail(B200_ESHAPE, "b200_tile_attn: %zu bytes of shared memory", smem);
  auto kern = tile_attn_kernel<T, DK, DV, ALIAS, MODE, HALVES, CTAS>;
  if constexpr (P::kSplitRegs) {
    int regs = 0;
    if (const cudaError_t e = built_registers<T, DK, DV, ALIAS, MODE, HALVES, CTAS>(&regs); e != cudaSuccess) {
      cudaGetLastError();
      return fail(static_cast<int>(e), "b200_tile_attn: %s", cudaGetErrorString(e));
    }
    if (!P::enough(regs)) return fail(B200_EINVAL, "b200_tile_attn: built with %d registers per thread", regs);
  }
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  TileAttn B = A;
  CUtensorMap k_map{}, v_map{}, q_map{};
  // pages that divide a tile of keys, rows that start on 16 bytes
  B.boxes = A.block_size % 8 == 0 && kKeys % A.block_size == 0 && page_map<T>(&k_map, A.k_pool, DK, A.block_size) &&
            (ALIAS || (A.v_row % 8 == 0 && page_map<T>(&v_map, A.v_pool, A.v_row, A.block_size)));
  B.q_boxes = query_map<T>(&q_map, A, DK);
  B.n_tiles = n_tiles;
  constexpr int kMost = 65535;      // of a grid's second dimension
  for (B.tile0 = 0; B.tile0 < n_tiles; B.tile0 += kMost) {
    kern<<<dim3(A.G, std::min(kMost, n_tiles - B.tile0), n_splits), P::kNT, smem, stream>>>(B, k_map, v_map, q_map);
    if (int rc = check_launch("b200_tile_attn")) return rc;
  }
  return 0;
}

template <int DK, int DV, bool ALIAS>
struct Shape {
  static constexpr int dk = DK, dv = DV;
  static constexpr bool alias = ALIAS;
};
template <typename T>
int launch_shape(const TileAttn& A, int dk, int dv, bool alias, int rows, int n_tiles, int n_splits, cudaStream_t stream) {
  auto go = [&](auto shape, auto mode) {
    constexpr int DK = decltype(shape)::dk, DV = decltype(shape)::dv, MODE = decltype(mode)::value;
    if constexpr (!decltype(shape)::alias) {
      if (rows != kRows) return launch_tiles<T, DK, DV, false, MODE, 2, 1>(A, n_tiles, n_splits, stream);
      // one CTA per SM has registers for its scores and warps that rescale (4 heads over 1, plain, 5 x 1024: 25.4 us against 30.1 side by side; 8 over 2, 3 x
      // 550: 17.8 / 20.4); more CTAs than SMs hide each other's beginnings (4 over 1, 64 x 96: 10.7 / 14.6)
      if (static_cast<int64_t>(n_tiles) * A.G * n_splits > kNumSMs) return launch_tiles<T, DK, DV, false, MODE, 1, 2>(A, n_tiles, n_splits, stream);
    }
    return launch_tiles<T, DK, DV, decltype(shape)::alias, MODE, 1, 1>(A, n_tiles, n_splits, stream);
  };
  auto by_mode = [&](auto shape) {
    if constexpr (!decltype(shape)::alias) {
      if (A.bias_lut) return go(shape, std::integral_constant<int, kBiased>{});
    }
    return A.softcap > 0.f ? go(shape, std::integral_constant<int, kCapped>{}) : go(shape, std::integral_constant<int, kPlain>{});
  };
  if (!alias && dk == 128 && dv == 128) return by_mode(Shape<128, 128, false>{});
  if (!alias && dk == 64 && dv == 64) return by_mode(Shape<64, 64, false>{});
  if (alias && dk == 256 && dv == 256) return by_mode(Shape<256, 256, true>{});
  if (alias && dk == 320 && dv == 256) return by_mode(Shape<320, 256, true>{});
  return fail(B200_ESHAPE, "b200_tile_attn: head sizes %d / %d are not built", dk, dv);
}

}  // namespace

bool tile_attn_supported(int H, int G, int dk, int dv, bool alias, bool bias, int dtype) {
  if (dtype != B200_DTYPE_BF16 && dtype != B200_DTYPE_F16) return false;
  if (H <= 0 || G <= 0 || H % G || H / G > (bias ? 16 : kTileRows)) return false;
  if (alias) return !bias && dv == 256 && (dk == 256 || dk == 320);
  return dk == dv && (dk == 64 || dk == 128);
}

// 256 rows share a fetched key tile and its biases and take turns with the exponentials; 128 rows have shorter beginnings and less of the causal
// triangle to mask.  With biases or a cap 256 rows are ahead where heads share their keys and there is more than an SM's CTA and a half of 128 (16
// over 4, 8 x 2048: 206 / 242 us against 241 / 285; 6 x 300 .. 640: 24 / 27 against 28 / 32; but 4 over 1, 8 x 700: 27 against 21 of plain
// scores), 128 where they do not share (16 over 16, 8 x 700: 60 / 67 against 64 / 70; 64 x 96: 50 / 53 against 73 / 73).  Plain scores keep 128 rows:
// ahead for short portions (16 over 4, 128 / 256 rows: 32 x 512 84 / 91, 8 x 700 38 / 39; 16 over 16 95 / 111, 48 / 55), behind for long ones
// (16 over 4, 8 x 2048 188 / 184, 4 x 4000 314 / 297; 8 over 2 of 64, 8 x 2048 89 / 78), whose length the rule is not told.
// Pages that come row by row keep 256 rows from one round of CTAs on with biases or a cap, from three without (8 x 1000 tokens of 16 heads, pages
// of 24: 82 us against 94 when the line was drawn; 79 now).
int tile_attn_rows(int rep, int G, int dk, int n_tokens, bool heavy, bool boxes) {
  const int64_t ctas = static_cast<int64_t>(n_tokens) * rep / (2 * kTileRows) * G;      // of 256 rows
  const bool wide = boxes ? heavy && rep > 1 && 4 * ctas > 3 * kNumSMs : ctas >= (heavy ? 1 : 3) * kNumSMs;
  if (!wide || dk > 128) return kTileRows;
  const bool built = dk <= 64 ? wide_built<__nv_bfloat16, 64>() && wide_built<__half, 64>() : wide_built<__nv_bfloat16, 128>() && wide_built<__half, 128>();
  return built ? 2 * kTileRows : kTileRows;
}

// Keys are divided while the chip has room for more CTAs, a share being worth its part of the merge: three tiles of 64 keys where
// few rows are merged, eight otherwise.  Room is one CTA per SM or two, whose walks are half as slow again each; which, by the sum of a walk and
// its merge, in microseconds of a key tile: 0.7 ns for every share of a live row of 128 values, 2 for the launch.  Full tiles keep an SM each (16
// heads over 4, 1 x 1024: undivided 18 us, in two 52; 8 x 64 tokens of 4 heads with keys of their own behind 1000: 4 shares 20.8, 5, two per SM,
// 23.5) unless the walks are long (8 over 2 of 64, 1000 behind 6000: 2 shares 71, 4 59); few tokens are soon merged (4 heads with keys of their own, 20
// x 4 tokens behind 3000: undivided 57, 3 shares 42; 8 x 2 behind 8000: 4 shares 45, 9 39).  Over 490 shapes and modes 0.4 % behind the better of the two.
int tile_attn_splits(int n_tiles, int key_tiles, int G, int dk, int rows, int64_t live_rows) {
  const int64_t ctas = static_cast<int64_t>(n_tiles) * G;
  auto divide = [&](int64_t room) {
    if (ctas <= 0 || ctas * 2 > room) return 1;
    const int share = ctas * rows <= 4096 ? 3 : 8;
    return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>({16, room / ctas, key_tiles / share})));
  };
  const int64_t live = std::min(live_rows, ctas * rows);      // (the call's tokens may have other portions among them)
  auto cost = [&](int splits) {
    const double walk = static_cast<double>(key_tiles) / splits * (splits * ctas > kNumSMs ? 1.5 : 1.0);
    return splits == 1 ? walk : walk + 2.0 + 0.0007 * static_cast<double>(live) * splits * dk / 128;
  };
  const int one_per_sm = divide(kNumSMs);
  if (rows != kTileRows || dk > 128) return one_per_sm;
  const int two_per_sm = divide(2 * kNumSMs);
  return cost(two_per_sm) < cost(one_per_sm) ? two_per_sm : one_per_sm;
}

int tile_attn_launch(const TileAttn& A, int dk, int dv, bool alias, int rows, int n_tiles, int n_splits, int dtype, cudaStream_t stream) {
  return dtype == B200_DTYPE_BF16 ? launch_shape<__nv_bfloat16>(A, dk, dv, alias, rows, n_tiles, n_splits, stream)
                                  : launch_shape<__half>(A, dk, dv, alias, rows, n_tiles, n_splits, stream);
}

}  // namespace b200
