// FP32 distance tests of neighbour candidates, B = 8 or 16 consecutive sorted slots at a time.
//
// The sorted FP32 positions are stored in chunks of four slots, {x0..x3, y0..y3, z0..z3} (2D:
// without z), so one 16-byte load fetches one coordinate of four consecutive candidates and its
// halves are operand pairs of the packed FP32 instructions (add / mul / fma.rn.f32x2: two IEEE
// operations per instruction, each rounded like the scalar one).  Against an array of {x, y, z, w}
// records this takes 3 loads in place of 4 per four candidates and half the arithmetic
// instructions.  A batch starts at a multiple of four slots; slots before a row's first or after
// its last are masked out by the caller.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pg_f32x2.cuh"

namespace pg {

// min(m, |a|, |b|); NaNs are ignored.
__device__ __forceinline__ float min3_abs(float m, float a, float b) {
  return fminf(m, fminf(fabsf(a), fabsf(b)));
}

// Floats of the chunked FP32 positions of n slots, with the chunks a batch may read past the last
// slot (it starts at or before its row's last slot, rounded down to a multiple of 4).
__host__ __device__ inline size_t chunked_floats(size_t n, int dim) { return ((n + 3) / 4 + 3) * 4 * dim; }

template <int DIM>
__device__ __forceinline__ size_t chunk_index(uint32_t k) {
  return (size_t)(k / 4) * (4 * DIM) + (k & 3u);
}

// The FP32 position of slot k.
template <int DIM>
__device__ __forceinline__ float4 pf_at(const float* pf, uint32_t k) {
  const float* p = pf + chunk_index<DIM>(k);
  return make_float4(p[0], p[4], DIM == 3 ? p[8] : 0.f, 0.f);
}

template <int DIM>
__device__ __forceinline__ void pf_store(float* pf, uint32_t k, float x, float y, float z) {
  float* p = pf + chunk_index<DIM>(k);
  p[0] = x;
  p[4] = y;
  if (DIM == 3) p[8] = z;
}

// The coordinates of one batch.
template <int DIM, int B>
struct Batch {
  ulonglong2 v[B / 4][DIM];
  __device__ __forceinline__ void load(const float* pf, uint32_t t) {  // t a multiple of 4
    const ulonglong2* p = (const ulonglong2*)pf + (size_t)(t / 4) * DIM;
#pragma unroll
    for (int i = 0; i < B / 4; ++i)
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[i][d] = __ldg(p + i * DIM + d);
  }
};

// Bounds on the FP32 r^2 of a candidate of a target at p (FP32 positions rounded from f64; reach: at
// least the support radius in FP32):  |x_j - x_i| < reach in f64  =>  r^2 < outer_threshold, and
// r^2 < inner_threshold  =>  |x_j - x_i| < reach in f64.  delta bounds the rounding of the
// positions and of the FP32 arithmetic with a generous factor.
__device__ __forceinline__ float outer_threshold(float reach, const float4& p) {
  const float M = fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fabsf(p.z)) + reach;
  const float delta = 2.384185791015625e-07f * (2.f * M + reach);  // 4u (2M + reach)
  const float rr = reach + 2.f * delta;
  return rr * rr * 1.0000153f;
}
__device__ __forceinline__ float inner_threshold(float reach, const float4& p) {
  const float M = fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fabsf(p.z)) + reach;
  const float delta = 2.384185791015625e-07f * (2.f * M + reach);
  const float rr = fmaxf(reach - 2.f * delta, 0.f);
  return rr * rr * 0.9999847f;
}

// The FP32 test of one target against thresholds on r^2.  With
// s = r^2 / mid - 1 (RATIO) or r^2 - mid (exact sign), a candidate is inside when s < 0.  Candidates
// with |r^2 s| <= tol are not decided by FP32 (r^2 close to mid, or zero, or tiny against it).
struct Screen {
  f2 nx, ny, nz;  // minus the target's position
  f2 a, b;        // RATIO: s = r^2 a + b; otherwise s = r^2 + b
  float tol;
};

// Thresholds for a decision in f64 (or by a superset): inside for certain below thr_lo, outside for
// certain from thr on.  Every r^2 in [thr_lo, thr) has |r^2 / mid - 1| <= w, with the rounding of
// 1 / mid and of the FMA added to w, hence r^2 |s| <= thr w = tol; and where r^2 |s| > tol, r^2 is
// not zero and either lies beyond thr (s > 0) or has |s| > w.  Where a square, the middle or its
// reciprocal may leave the normal FP32 range, every candidate is left undecided.
__device__ __forceinline__ void screen_band(Screen& s, float thr_lo, float thr) {
  const float mid = 0.5f * (thr_lo + thr);
  const float inv = 1.0f / mid;
  const float w = 0.5f * (thr - thr_lo) * inv + 4.76837158203125e-07f;  // + 8u
  s.a = f2_dup(inv);
  s.b = f2_dup(-1.0f);
  s.tol = thr > 1e-30f && thr < 1e37f ? thr * w * 1.00001f : __int_as_float(0x7f800000);
}

// Threshold compared exactly (IEEE r^2 < thr); only r^2 = 0 (or an underflow) is left undecided.
__device__ __forceinline__ void screen_exact(Screen& s, float thr) {
  s.a = 0ull;
  s.b = f2_dup(-thr);
  s.tol = 0.f;
}

__device__ __forceinline__ void screen_target(Screen& s, const float4& p) {
  s.nx = f2_dup(-p.x);
  s.ny = f2_dup(-p.y);
  s.nz = f2_dup(-p.z);
}

// Decisions for the B candidates of a batch, candidate b at bit B - 1 - b: the sign bits of
// s (inside), and in `open` the candidates FP32 does not decide (masked-out ones included).
// CONTRACT: r^2 with fused multiply-adds; otherwise (x^2 + y^2) + z^2, each operation rounded.
template <int DIM, int B, bool CONTRACT, bool RATIO>
__device__ __forceinline__ unsigned screen_batch(const Batch<DIM, B>& C, const Screen& S, unsigned& open) {
  unsigned in = 0;
  float q[B], m = 3.402823466e38f;
#pragma unroll
  for (int i = 0; i < B / 2; ++i) {
    const int c = i / 2;
    const f2 dx = f2_add(i & 1 ? C.v[c][0].y : C.v[c][0].x, S.nx), dy = f2_add(i & 1 ? C.v[c][1].y : C.v[c][1].x, S.ny);
    f2 r2 = CONTRACT ? f2_mul(dx, dx) : f2_mul_rn(dx, dx);
    r2 = CONTRACT ? f2_fma(dy, dy, r2) : f2_add(r2, f2_mul_rn(dy, dy));
    if (DIM == 3) {
      const f2 dz = f2_add(i & 1 ? C.v[c][DIM - 1].y : C.v[c][DIM - 1].x, S.nz);
      r2 = CONTRACT ? f2_fma(dz, dz, r2) : f2_add(r2, f2_mul_rn(dz, dz));
    }
    const f2 s = RATIO ? f2_fma(r2, S.a, S.b) : f2_add(r2, S.b);
    const float2 sv = f2_split(s), qv = f2_split(f2_mul(r2, s));
    in = __funnelshift_l(__float_as_uint(sv.x), in, 1);  // in = 2 in + sign bit
    in = __funnelshift_l(__float_as_uint(sv.y), in, 1);
    m = min3_abs(m, qv.x, qv.y);
    q[2 * i] = qv.x;
    q[2 * i + 1] = qv.y;
  }
  open = 0;
  if (!(m > S.tol)) {
#pragma unroll
    for (int b = 0; b < B; ++b) open = 2 * open + (fabsf(q[b]) > S.tol ? 0u : 1u);
  }
  return in;
}

}  // namespace pg
