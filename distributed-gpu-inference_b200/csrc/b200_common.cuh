// Shared helpers for the sm_100a paged-KV kernels: error plumbing for the C ABI, dtype traits, vector
// load/store wrappers.  Nothing here allocates or synchronises.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/b200_kv.h"

namespace b200 {

// ---- error plumbing ---------------------------------------------------------------------------------
char* last_error_buf();  // thread-local, defined in b200_abi.cu
constexpr int kErrBufLen = 512;

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buf(), kErrBufLen, fmt, ap);
  va_end(ap);
  return code;
}

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(static_cast<int>(e), "%s: %s", what, cudaGetErrorString(e));
  return 0;
}

inline int dtype_size(int dtype) {
  switch (dtype) {
    case B200_DTYPE_F16:
    case B200_DTYPE_BF16:
      return 2;
    case B200_DTYPE_F32:
      return 4;
    default:
      return 0;
  }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ---- device helpers ---------------------------------------------------------------------------------
template <typename T>
struct Cvt;
template <>
struct Cvt<float> {
  static __device__ __forceinline__ float to_f32(float x) { return x; }
  static __device__ __forceinline__ float from_f32(float x) { return x; }
};
template <>
struct Cvt<__half> {
  static __device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half from_f32(float x) { return __float2half_rn(x); }
};
template <>
struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 from_f32(float x) { return __float2bfloat16_rn(x); }
};

// streaming 16-byte global load / store: data that is touched once should not displace L1 lines
__device__ __forceinline__ int4 ld_stream16(const void* p) {
  int4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}
__device__ __forceinline__ void st_stream16(void* p, const int4& v) {
  asm volatile("st.global.L1::no_allocate.v4.s32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 1 / (1 + e^-z) as n / d with t = e^-|z|, d = 1 + t in [1, 2], n = 1 or t.  The quotient is an approximate reciprocal's, put right by one
// Newton step on its remainder, which counts what d lost in its rounding (Dekker's sum); d needs no care for overflow, so there is no branch between the elements of a row, whose chains then
// overlap.  (A general division branches: row kernels with one sigmoid per element were bound by it, with the wider pieces 52 -> 35 us for 16384 x 8 gated rows of 128, bf16.)  Infinities give 0 and 1, NaN NaN.
// z times this over 2^20 points of -80 .. 80 against 64 bits: largest relative error 2.11e-7, mean 2.25e-8 (by division 2.25e-7, 2.56e-8).
__device__ __forceinline__ float row_logistic(float z) {
  const float t = expf(-fabsf(z));
  const float d = 1.0f + t, n = z < 0.f ? t : 1.0f;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = n * r, lost = t - (d - 1.0f);
  return fmaf(fmaf(-q, lost, fmaf(-q, d, n)), r, q);
}

// The same of two numbers, the same bits: what is no exponential or reciprocal takes both at once.
__device__ __forceinline__ float2 row_logistic2(float x, float y) {
  using Pair = unsigned long long;
  auto pair = [](float a, float b) {
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
  };
  auto mul = [](Pair a, Pair b) {
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
  };
  auto add = [](Pair a, Pair b) {
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
  };
  auto fma = [](Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
  };
  const float tx = expf(-fabsf(x)), ty = expf(-fabsf(y));
  const Pair t = pair(tx, ty), d = add(pair(1.0f, 1.0f), t), n = pair(x < 0.f ? tx : 1.0f, y < 0.f ? ty : 1.0f);
  float dx, dy, rx, ry;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(dx), "=f"(dy) : "l"(d));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"(dx));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ry) : "f"(dy));
  const Pair r = pair(rx, ry), q = mul(n, r), minus_q = mul(n, pair(-rx, -ry));
  const Pair lost = fma(add(d, pair(-1.0f, -1.0f)), pair(-1.0f, -1.0f), t);      // t - (d - 1): the product is exact
  const Pair s = fma(fma(minus_q, lost, fma(minus_q, d, n)), r, q);
  float2 out;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(out.x), "=f"(out.y) : "l"(s));
  return out;
}

constexpr int kNumSMs = 148;  // B200
constexpr int kMaxSmem = 227 * 1024;   // a CTA's shared memory: the limit to set where launches of one kernel differ in size (another
                                       // thread's smaller one between setting it and the launch would make that fail)

}  // namespace b200
