// Pairs of 32-bit floats in one 64-bit register and the instructions that work on both at once (fma.rn.f32x2 and
// relatives: two IEEE operations, rounded like the scalar ones, for one issue slot).
#pragma once
#include <stdint.h>

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 f2_pack(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ f32x2 f2_both(float x) { return f2_pack(x, x); }
__device__ __forceinline__ void f2_unpack(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// (x + y) + (z + w) of two pairs
__device__ __forceinline__ float f2_sum4(f32x2 xy, f32x2 zw) {
  float x, y, z, w;
  f2_unpack(xy, x, y);
  f2_unpack(zw, z, w);
  return (x + y) + (z + w);
}
// Four floats (16-byte aligned, shared or global memory) as two pairs.
__device__ __forceinline__ void f2_load4(const float* p, f32x2& xy, f32x2& zw) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  xy = v.x;
  zw = v.y;
}
