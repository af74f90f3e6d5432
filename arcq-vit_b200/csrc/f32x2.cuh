// Two fp32 values per instruction, and pairs of 16-bit values to and from them.
//
// A packed add, mul or fma takes the pipe two cycles, as two scalar ones do, and one issue slot instead of two (measured: 2.00 and 1.01
// cycles a warp instruction on a scheduler).  lop3, min / max of three, conversions between fp16 and fp32 and half2 arithmetic take
// their pipe two cycles as well.
#pragma once
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace arcq {

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// A packed mul whose result feeds a packed add is contracted into one fma by the assembler, .rn on both notwithstanding (one
// rounding instead of two: a scale came out one unit in the last place off).  Where that matters, mul2_rn adds a -0 that
// the compiler cannot see (GroupQuantParams::nz), which leaves every product as it is.
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2_rn(f32x2 a, f32x2 b, f32x2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f32x2 fma2_down(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float min3_abs(float m, float a, float b) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(m), "f"(fabsf(a)), "f"(fabsf(b)));
  return d;
}

template <typename T> __device__ __forceinline__ f32x2 sixteen_to_pair(uint32_t w);
template <> __device__ __forceinline__ f32x2 sixteen_to_pair<__half>(uint32_t w) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  return pack2(f.x, f.y);
}
template <> __device__ __forceinline__ f32x2 sixteen_to_pair<__nv_bfloat16>(uint32_t w) {
  return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <typename T> __device__ __forceinline__ uint32_t pair_to_sixteen(f32x2 v);
template <> __device__ __forceinline__ uint32_t pair_to_sixteen<__half>(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pair_to_sixteen<__nv_bfloat16>(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

}  // namespace arcq
