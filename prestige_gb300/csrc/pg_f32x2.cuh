// Packed FP32: two floats in a 64-bit register pair and the f32x2 instructions on them.  Each half is rounded
// like the scalar instruction; the FMA pipe takes as long as for two scalar instructions, but they
// need one issue slot.
#pragma once
#include <cuda_runtime.h>

namespace pg {

typedef unsigned long long f2;  // two floats: .lo is the low word

__device__ __forceinline__ f2 f2_make(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 f2_dup(float v) { return f2_make(v, v); }
__device__ __forceinline__ float2 f2_split(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// The product rounded on its own: mul.rn.f32x2 may be fused with an addition that takes its result (measured:
// a product plus a product is), the scalar instructions are not.
__device__ __forceinline__ f2 f2_mul_rn(f2 a, f2 b) {
  const float2 x = f2_split(a), y = f2_split(b);
  return f2_make(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y));
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// -v (folded into the instruction that takes it; an exclusive or of the sign bits is not)
__device__ __forceinline__ f2 f2_neg(f2 v) {
  const float2 s = f2_split(v);
  return f2_make(-s.x, -s.y);
}

}  // namespace pg
