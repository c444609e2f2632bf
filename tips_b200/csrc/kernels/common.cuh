// Shared helpers of the sm_100a kernel library: error plumbing for the
// extern "C" launchers, dtype codes, vector load/store helpers.
//
// Every launcher returns 0 on success or a negative code and leaves a message
// retrievable with tipsk_last_error(); none of them allocates device memory
// unless its name says so, and all of them launch on the stream they are given.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace tipsk {

// Values match tips::Datatype on the host side.
enum DType : int32_t { kF32 = 0, kF64 = 1, kI32 = 2, kI64 = 3, kI8 = 4, kU8 = 5, kBF16 = 6, kF16 = 7 };

inline size_t DTypeSize(int32_t dt) {
  switch (dt) {
    case kF32: case kI32: return 4;
    case kF64: case kI64: return 8;
    case kI8: case kU8: return 1;
    case kBF16: case kF16: return 2;
    default: return 0;
  }
}

std::string& LastError();
int SetError(int code, const std::string& msg);

#define TIPSK_CUDA(expr)                                                                          \
  do {                                                                                            \
    cudaError_t _e = (expr);                                                                      \
    if (_e != cudaSuccess)                                                                        \
      return ::tipsk::SetError(-7, std::string(#expr) + ": " + cudaGetErrorString(_e));           \
  } while (0)

#define TIPSK_LAUNCH_CHECK()                                                                      \
  do {                                                                                            \
    cudaError_t _e = cudaGetLastError();                                                          \
    if (_e != cudaSuccess)                                                                        \
      return ::tipsk::SetError(-7, std::string("kernel launch failed: ") + cudaGetErrorString(_e)); \
  } while (0)

#define TIPSK_REQUIRE(cond, msg)                         \
  do {                                                   \
    if (!(cond)) return ::tipsk::SetError(-2, (msg));    \
  } while (0)

inline int CeilDiv(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }

// Number of SMs of the current device (cached).
int NumSMs();

// ---- device-side conversions ------------------------------------------------
template <typename T>
__device__ __forceinline__ float ToFloat(T v);
template <>
__device__ __forceinline__ float ToFloat<float>(float v) { return v; }
template <>
__device__ __forceinline__ float ToFloat<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float ToFloat<__half>(__half v) { return __half2float(v); }

template <typename T>
__device__ __forceinline__ T FromFloat(float v);
template <>
__device__ __forceinline__ float FromFloat<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 FromFloat<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half FromFloat<__half>(float v) { return __float2half_rn(v); }

// ---- two fp32 values per instruction (fma.rn.f32x2 and its relatives) --------
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 MakeF2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 SplitF2(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 Fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 Mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 Both(float a) { return MakeF2(a, a); }
__device__ __forceinline__ F2 Exp2Fast(F2 a) {
  float2 x = SplitF2(a);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(x.x));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(x.y));
  return MakeF2(x.x, x.y);
}
__device__ __forceinline__ F2 RcpFast(F2 a) {
  float2 x = SplitF2(a);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(x.x));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(x.y));
  return MakeF2(x.x, x.y);
}

// erfc(z) / exp(-z^2) for z = |v| / sqrt(2) by the rational approximation a1 t + ... + a5 t^5, t = 1 / (1 + p z)
// (Abramowitz and Stegun, 7.1.26: absolute error of erf < 1.5e-7), and exp(-z^2), of two values at once.  For results
// that are rounded to 16 bits next: one exponential and one reciprocal where erff takes two divergent branches.  Error of the
// bf16 GELU against 64 bits (relative 2-norm, with 0.5 v (1 + erff) : like this): normally distributed v 1.6645e-3 : 1.6645e-3,
// v in -3..0 1.7087e-3 : 1.7087e-3, -4..-3 1.5916e-3 : 1.5944e-3, and beyond, where 1 + erff cancels, -6..-4 2.22e-3 : 1.69e-3.
__device__ __forceinline__ void ErfcParts2(F2 v, F2* poly, F2* gauss) {
  const float2 s = SplitF2(v);
  const F2 z = Mul2(MakeF2(fabsf(s.x), fabsf(s.y)), Both(0.70710678118654752f));
  const F2 t = RcpFast(Fma2(z, Both(0.3275911f), Both(1.f)));
  F2 q = Fma2(t, Both(1.061405429f), Both(-1.453152027f));
  q = Fma2(t, q, Both(1.421413741f));
  q = Fma2(t, q, Both(-0.284496736f));
  q = Fma2(t, q, Both(0.254829592f));
  *poly  = Mul2(t, q);
  *gauss = Exp2Fast(Mul2(Mul2(z, z), Both(-1.4426950408889634f)));
}
// GELU v * Phi(v): no cancellation for negative v, where Phi is half of erfc itself.
__device__ __forceinline__ F2 Gelu2(F2 v) {
  F2 poly, gauss;
  ErfcParts2(v, &poly, &gauss);
  const F2 tail = Mul2(Mul2(poly, gauss), Both(0.5f));       // Phi(-|v|)
  const float2 lo = SplitF2(tail), hi = SplitF2(Fma2(tail, Both(-1.f), Both(1.f))), s = SplitF2(v);
  return Mul2(v, MakeF2(s.x < 0.f ? lo.x : hi.x, s.y < 0.f ? lo.y : hi.y));
}
// Its derivative Phi(v) + v * phi(v).
__device__ __forceinline__ F2 GeluGrad2(F2 v) {
  F2 poly, gauss;
  ErfcParts2(v, &poly, &gauss);
  const F2 tail = Mul2(Mul2(poly, gauss), Both(0.5f));
  const float2 lo = SplitF2(tail), hi = SplitF2(Fma2(tail, Both(-1.f), Both(1.f))), s = SplitF2(v);
  const F2 cdf = MakeF2(s.x < 0.f ? lo.x : hi.x, s.y < 0.f ? lo.y : hi.y);
  return Fma2(Mul2(v, Both(0.3989422804014327f)), gauss, cdf);
}

// 16-byte vector of T.
template <typename T>
struct alignas(16) Vec16 {
  static constexpr int kN = 16 / sizeof(T);
  T v[kN];
};

template <typename T>
__device__ __forceinline__ Vec16<T> LoadVec(const T* p) {
  return *reinterpret_cast<const Vec16<T>*>(p);
}
template <typename T>
__device__ __forceinline__ void StoreVec(T* p, const Vec16<T>& v) {
  *reinterpret_cast<Vec16<T>*>(p) = v;
}

__device__ __forceinline__ float WarpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float WarpMax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace tipsk
