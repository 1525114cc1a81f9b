// The packed FP32 helpers (prestige_gb300/csrc/pg_f32x2.cuh, the df2 operations of pg_arith.cuh and the
// candidate screen of pg_candidates.cuh) against the scalar operations, bit for bit.  Run by
// tests/test_gpu_packed.py.
//   df2_*, dfacc_add_prod2   each half equals the scalar double-word operation
//   screen_batch (IEEE)      decides as r^2 = (dx dx + dy dy) + dz dz with every operation rounded, on
//                            positions whose r^2 lies within a few units of the threshold
#include <cstdint>
#include <cstdio>

#include "../../prestige_gb300/csrc/pg_arith.cuh"
#include "../../prestige_gb300/csrc/pg_candidates.cuh"

using namespace pg;

__device__ uint32_t next(uint32_t& s) {  // xorshift32 (Marsaglia 2003)
  s ^= s << 13;
  s ^= s >> 17;
  s ^= s << 5;
  return s;
}
__device__ float rnd(uint32_t& s) {
  const uint32_t m = next(s) & 0x807fffffu;
  return __uint_as_float(m | ((120u + next(s) % 14u) << 23));
}
__device__ df rnd_df(uint32_t& s) {
  const float h = rnd(s), e = __uint_as_float((next(s) & 0x807fffffu) | (101u << 23));
  return fast_two_sum(h, h * e);
}
__device__ bool ne(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
__device__ bool ne(df2 v, df a, df b) {
  const df x = df2_first(v), y = df2_second(v);
  return ne(x.hi, a.hi) || ne(x.lo, a.lo) || ne(y.hi, b.hi) || ne(y.lo, b.lo);
}

enum { kMul, kMulF, kDiv, kAddRaw, kSub, kSubClose, kAcc, kScreen2, kScreen3, kTests };

template <int DIM>
__device__ void screen(uint32_t& s, unsigned long long* bad) {
  __align__(16) float pf[2 * 4 * DIM];
  float4 p = make_float4(rnd(s), rnd(s), DIM == 3 ? rnd(s) : 0.f, 0.f);
  float x[8][3];
  float thr = 0.f;
  for (int b = 0; b < 8; ++b) {
    for (int d = 0; d < 3; ++d) x[b][d] = rnd(s);
    const float d0 = __fsub_rn(p.x, x[b][0]), d1 = __fsub_rn(p.y, x[b][1]), d2 = __fsub_rn(p.z, x[b][2]);
    float r2 = __fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1));
    if (DIM == 3) r2 = __fadd_rn(r2, __fmul_rn(d2, d2));
    if (b == 0) thr = __uint_as_float(__float_as_uint(r2) + next(s) % 3u - 1u);
    if (b) {  // near the first one: coordinates exchanged, signs changed, a last bit moved
      const int o = next(s) % DIM;
      for (int d = 0; d < DIM; ++d) {
        const float q = d == 0 ? p.x : d == 1 ? p.y : p.z;
        const int c = (d + o) % DIM;
        const float qc = c == 0 ? p.x : c == 1 ? p.y : p.z;
        x[b][d] = q + (next(s) & 1 ? 1.f : -1.f) * (x[0][c] - qc);
        if (next(s) % 4 == 0) x[b][d] = __uint_as_float(__float_as_uint(x[b][d]) + 1u);
      }
    }
    pf_store<DIM>(pf, b, x[b][0], x[b][1], x[b][2]);
  }
  Screen S;
  screen_target(S, p);
  screen_exact(S, thr);
  Batch<DIM, 8> B;
  for (int i = 0; i < 2; ++i)
    for (int d = 0; d < DIM; ++d) B.v[i][d] = *(const ulonglong2*)(pf + (i * DIM + d) * 4);
  unsigned open;
  const unsigned in = screen_batch<DIM, 8, false, false>(B, S, open);
  for (int b = 0; b < 8; ++b) {
    const float d0 = __fsub_rn(p.x, x[b][0]), d1 = __fsub_rn(p.y, x[b][1]), d2 = __fsub_rn(p.z, x[b][2]);
    float r2 = __fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1));
    if (DIM == 3) r2 = __fadd_rn(r2, __fmul_rn(d2, d2));
    if (!(open >> (7 - b) & 1u) && (in >> (7 - b) & 1u) != (r2 < thr ? 1u : 0u))
      atomicAdd(bad + (DIM == 2 ? kScreen2 : kScreen3), 1ull);
  }
}

__global__ void check(unsigned long long* bad) {
  uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + 12345u;
  if (!s) s = 1;
  for (int i = 0; i < 200; ++i) {
    const df x = rnd_df(s), y = rnd_df(s), x2 = rnd_df(s), y2 = rnd_df(s);
    const df2 X = df2_pair(x, x2), Y = df2_pair(y, y2);
    const float f = rnd(s), f2nd = rnd(s);
    if (ne(df2_mul(X, Y), df_mul(x, y), df_mul(x2, y2))) atomicAdd(bad + kMul, 1ull);
    if (ne(df2_mul_f(X, f2_make(f, f2nd)), df_mul_f(x, f), df_mul_f(x2, f2nd))) atomicAdd(bad + kMulF, 1ull);
    if (ne(df2_div(X, Y), df_div(x, y), df_div(x2, y2))) atomicAdd(bad + kDiv, 1ull);
    if (ne(df2_add_raw(X, Y), df_add_raw(x, y), df_add_raw(x2, y2))) atomicAdd(bad + kAddRaw, 1ull);
    if (ne(df2_sub(X, Y), df_sub(x, y), df_sub(x2, y2))) atomicAdd(bad + kSub, 1ull);
    if (ne(df2_sub_close(X, Y), df_sub_close(x, y), df_sub_close(x2, y2))) atomicAdd(bad + kSubClose, 1ull);
    dfacc a, b;
    a.hi = b.hi = f;
    a.lo = b.lo = f * 1e-8f;
    dfacc_add_prod2(a, X, Y);
    dfacc_add_prod(b, x, y);
    dfacc_add_prod(b, x2, y2);
    if (ne(a.hi, b.hi) || ne(a.lo, b.lo)) atomicAdd(bad + kAcc, 1ull);
    screen<2>(s, bad);
    screen<3>(s, bad);
  }
}

int main() {
  unsigned long long* bad;
  if (cudaMallocManaged(&bad, kTests * 8) != cudaSuccess) return 2;
  for (int i = 0; i < kTests; ++i) bad[i] = 0;
  check<<<512, 256>>>(bad);
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    fprintf(stderr, "%s\n", cudaGetErrorString(e));
    return 2;
  }
  const char* name[kTests] = {"df2_mul", "df2_mul_f", "df2_div", "df2_add_raw", "df2_sub", "df2_sub_close",
                              "dfacc_add_prod2", "screen 2D", "screen 3D"};
  int rc = 0;
  for (int i = 0; i < kTests; ++i)
    if (bad[i]) {
      fprintf(stderr, "%s: %llu differ\n", name[i], bad[i]);
      rc = 1;
    }
  return rc;
}
