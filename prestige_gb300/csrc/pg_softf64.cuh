// Correctly rounded f64 division, square root and multiplication on the integer and FP32 pipes.
//
// GB300 issues FP64 at 1/64 of the FP32 rate, so a division or square root in FP64 instructions
// (about 9 and 10 FP64 operations by measured throughput) occupies its pipe as long as about 600
// FP32 or 300 integer instructions would occupy theirs.  These take about 50 instructions and no FP64
// (per clock and SM: 1.32 divisions against 0.21, 1.46 roots each followed by an addition against 0.19):
//   1. the quotient (or root) Q of the 53-bit significands as an integer, from an FP32
//      approximation corrected once with its FP32 residual: off by less than 2^9 units
//   2. the exact remainder of that integer, R = A - Q B (or X - Q^2), in 64-bit integers modulo 2^64
//   3. the rest of the quotient d = R / B (or R / 2Q) in FP32, so Q + rint(d) is the correctly rounded
//      result unless d lies within its own error of a rounding boundary
// The result is the IEEE one, bit for bit; what step 3 does not decide (about one operand pair in
// 10^4), zeros, subnormals, infinities, NaNs and results outside the normal range take the hardware
// operation, out of line.  Newton's iteration for the approximations; the rounding decided on the
// exact remainder as in Markstein, IBM J. Res. Dev. 34 (1990).
//
// Bounds, in units of the last place of Q.  Step 1: the reciprocal after its Newton step is within
// 2^-23 (relative), so q0 is within 2^-22 and its residual r below 2^-20; the roundings of r
// (three, each 2^-24 r) and of q1 = r t leave less than 2^-43.5, about 360 units (the root's
// quadratic term adds 2^-45); a model with seeds at twice their documented error reaches 302.  So
// |R| < 2^63, and the signed 64-bit remainder is exact.  Step 3: leaving out the low word of R, 2^-20;
// reciprocal, truncated divisor, conversion and products, 2^-21.2 |d|.
#pragma once
#include <cuda_runtime.h>

namespace pg {

static __device__ __noinline__ double div_f64_call(double a, double b) { return __ddiv_rn(a, b); }
static __device__ __noinline__ double sqrt_f64_call(double x) { return __dsqrt_rn(x); }
// (inline, the compiler multiplies always and selects)
static __device__ __noinline__ double mul_f64_call(double a, double b) { return __dmul_rn(a, b); }

// d, with m = fl(d + 1.5 2^23), is far enough from a rounding boundary: |d - rint(d)| + 2^-21 |d| < 1/2 -
// 2^-19, and |d| < 512.
__device__ __forceinline__ bool soft_sure(float d, float m) {
  const float frac = fabsf(__fsub_rn(d, __fsub_rn(m, 12582912.0f)));
  return __fmaf_rn(fabsf(d), 4.76837158203125e-07f, frac) < 0.499998f && fabsf(d) < 512.0f;
}

// a / b, rounded to nearest even.
__device__ __forceinline__ double soft_div(double a, double b) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  const unsigned ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  const unsigned am = ah & 0xfffffu, bm = bh & 0xfffffu;
  // significands in [1, 2); the dividend doubled where it is the smaller, so the quotient is in [1, 2)
  const bool less = am < bm || (am == bm && al < bl);
  const unsigned eq = ea - eb + (less ? 1022u : 1023u);
  const float bf = __uint_as_float(0x3f800000u | __funnelshift_l(bl, bm, 3));
  const float af = __uint_as_float((less ? 0x40000000u : 0x3f800000u) | __funnelshift_l(al, am, 3));
  const float bt = (float)(int)(bl & 0x1fffffffu) * 2.220446049250313e-16f;                         // 2^-52
  const float at = (float)(int)(al & 0x1fffffffu) * (less ? 4.440892098500626e-16f : 2.220446049250313e-16f);
  float t;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(bf));
  t = __fmaf_rn(t, __fmaf_rn(-bf, t, 1.0f), t);
  const float q0 = fminf(fmaxf(__fmul_rn(af, t), 1.0f), 2.0f);
  const float r = __fadd_rn(__fmaf_rn(-q0, bf, af), __fmaf_rn(-q0, bt, at));
  const int q1 = __float2int_rn(__fmul_rn(r, __fmul_rn(t, 4503599627370496.0f)));  // 2^52
  const unsigned u = __float_as_uint(q0) - 0x3f000000u;                             // q0 2^23
  const unsigned long long q = ((unsigned long long)u << 29) + (unsigned long long)(long long)q1;
  const unsigned ql = (unsigned)q, qh = (unsigned)(q >> 32);
  const unsigned p = __umulhi(ql, bl) + ql * (bm | 0x100000u) + qh * bl;  // bits 32 .. 63 of Q B
  const int rem = (int)((al << (less ? 21 : 20)) - p);
  const float d = __fmul_rn((float)rem, __fmul_rn(t, 9.5367431640625e-07f));  // 2^-20
  const float m = __fadd_rn(d, 12582912.0f);                                  // 1.5 2^23: rint(d) in the low bits
  const bool sure = soft_sure(d, m) && ea - 1u < 2046u && eb - 1u < 2046u && eq - 1u < 2046u;
  if (!sure) return div_f64_call(a, b);
  const unsigned long long res = q + (unsigned long long)(long long)(__float_as_int(m) - 0x4b400000);
  const unsigned hi = (unsigned)(res >> 32) + ((eq - 1u) << 20);  // the leading bit of Q adds the 1
  return __hiloint2double((int)(hi | ((ah ^ bh) & 0x80000000u)), (int)(unsigned)res);
}

// sqrt(x), rounded to nearest even.
__device__ __forceinline__ double soft_sqrt(double x) {
  const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
  const unsigned e = xh >> 20;  // with the sign
  const bool even = !(e & 1u);  // odd binary exponent: significand in [2, 4)
  const unsigned xm = xh & 0xfffffu;
  const float f = __uint_as_float((even ? 0x40000000u : 0x3f800000u) | __funnelshift_l(xl, xm, 3));
  const float ft = (float)(int)(xl & 0x1fffffffu) * (even ? 4.440892098500626e-16f : 2.220446049250313e-16f);
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
  y = __fmaf_rn(__fmul_rn(0.5f, y), __fmaf_rn(-__fmul_rn(f, y), y, 1.0f), y);
  const float s0 = fminf(fmaxf(__fmul_rn(f, y), 1.0f), 2.0f);
  const float r = __fadd_rn(__fmaf_rn(-s0, s0, f), ft);
  const int s1 = __float2int_rn(__fmul_rn(r, __fmul_rn(y, 2251799813685248.0f)));  // 2^51
  const unsigned u = __float_as_uint(s0) - 0x3f000000u;                             // s0 2^23
  const unsigned long long s = ((unsigned long long)u << 29) + (unsigned long long)(long long)s1;
  const unsigned sl = (unsigned)s, sh = (unsigned)(s >> 32);
  const unsigned p = __umulhi(sl, sl) + sl * (2u * sh);  // bits 32 .. 63 of S^2
  const int rem = (int)((xl << (even ? 21 : 20)) - p);
  const float d = __fmul_rn((float)rem, __fmul_rn(y, 4.76837158203125e-07f));  // 2^-21
  const float m = __fadd_rn(d, 12582912.0f);
  const bool sure = soft_sure(d, m) && e - 1u < 2046u;
  if (!sure) return sqrt_f64_call(x);
  const unsigned long long res = s + (unsigned long long)(long long)(__float_as_int(m) - 0x4b400000);
  const unsigned hi = (unsigned)(res >> 32) + (((e + 1023u) >> 1) - 1u << 20);
  return __hiloint2double((int)hi, (int)(unsigned)res);
}

// a b, rounded to nearest even: the 106-bit product of the significands by four 32 x 32 bit multiplications,
// its leading 53 bits rounded on the bits below.  About 32 integer instructions against one FP64 one,
// that is about half of the FP64 pipe's time but on another pipe: for kernels whose FP64 pipe is full
// and whose other pipes are not.  Operands outside 2^-255 .. 2^257 (zeros among them) and possible ties
// take the FP64 instruction, out of line.
__device__ __forceinline__ double soft_mul(double a, double b) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  const unsigned am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
  // A in [2^52, 2^53) times B 2^11 in [2^63, 2^64): 2^115 .. 2^117, the high 64 bits h in [2^51, 2^53)
  const unsigned cl = bl << 11, ch = __funnelshift_l(bl, bm, 11);
  const unsigned long long m0 = (unsigned long long)al * cl;
  const unsigned long long m1 = (unsigned long long)am * cl + (unsigned)(m0 >> 32);
  const unsigned long long m2 = (unsigned long long)al * ch + (unsigned)m1;
  const unsigned long long h = (unsigned long long)am * ch + (unsigned)(m1 >> 32) + (unsigned)(m2 >> 32);
  const unsigned hl = (unsigned)h, hh = (unsigned)(h >> 32), below = (unsigned)m2;
  const unsigned s = ~(hh >> 20) & 1u;  // one bit to the left where h < 2^52
  const unsigned rh = __funnelshift_l(hl, hh, s), rl = __funnelshift_l(below, hl, s), rest = below << s;
  const unsigned long long r = (((unsigned long long)rh << 32) | rl) + (rest >> 31);
  // both exponents in 768 .. 1279 where neither difference has one of its two top bits set
  const bool in = ((((ah << 1) - 0x60000000u) | ((bh << 1) - 0x60000000u)) & 0xc0000000u) == 0;
  const unsigned e = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) - ((1023u << 20) + (s << 20));  // r has the leading bit
  const unsigned hi = ((unsigned)(r >> 32) + e) | ((ah ^ bh) & 0x80000000u);
  if (!in || rest == 0x80000000u) return mul_f64_call(a, b);
  return __hiloint2double((int)hi, (int)(unsigned)r);
}

}  // namespace pg
