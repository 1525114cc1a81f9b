// soft_div, soft_sqrt and soft_mul (prestige_gb300/csrc/pg_softf64.cuh) against the IEEE operations of
// the device (__ddiv_rn, __dsqrt_rn, __dmul_rn), bit for bit (NaNs as NaNs).  Run by tests/test_gpu_softf64.py.
//   random bit patterns (every exponent, subnormals, infinities, NaNs)
//   random significands with exponents near zero, and few-bit significands (exact quotients and roots)
//   operands whose quotient or root lies next to a representable number or next to a midpoint of two
//   zeros, ones, powers of two, the ends of the range
#include <cstdint>
#include <cstdio>

#include "../../prestige_gb300/csrc/pg_softf64.cuh"

using namespace pg;

__device__ uint64_t mix(uint64_t z) {  // splitmix64 (Steele, Lea, Flood 2014)
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__device__ double as_double(uint64_t b) { return __longlong_as_double((long long)b); }

__device__ double operand(int kind, uint64_t r) {
  const uint64_t frac = r & 0xfffffffffffffull, sign = r & 0x8000000000000000ull;
  switch (kind) {
    case 0: return as_double(r);                                            // any bits
    case 1: return as_double(sign | ((1013 + (r >> 52) % 21) << 52) | frac);  // around 1
    case 2: return as_double(sign | ((1013 + (r >> 52) % 21) << 52) | (frac & ~0ull << (r % 52)));  // few bits
    case 3: return as_double(sign | ((1013 + (r >> 52) % 21) << 52) | (frac | ((1ull << (r % 52)) - 1)) % (1ull << 52));
    default: {
      const double s[] = {0.0, -0.0, 1.0, -1.0, 2.0, 0.5, 4.0, 3.0, 1.0 / 3.0, 4.9e-324, -4.9e-324, 2.2250738585072014e-308,
                          2.225073858507201e-308, 1.7976931348623157e308, -1.7976931348623157e308, as_double(0x7ff0000000000000ull),
                          as_double(0xfff0000000000000ull), as_double(0x7ff8000000000000ull), as_double(0x3fefffffffffffffull),
                          as_double(0x3ff0000000000001ull), as_double(0x400fffffffffffffull), as_double(0x4010000000000001ull)};
      return s[r % (sizeof(s) / sizeof(s[0]))];
    }
  }
}

__device__ bool same(double a, double b) {
  return (a != a && b != b) || __double_as_longlong(a) == __double_as_longlong(b);
}

// bad[0..2]: mismatches of the division, the root and the product; ex: the first mismatching operands
__global__ void check(uint64_t seed, int iters, unsigned long long* bad, double* ex) {
  const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = 0; i < iters; ++i) {
    const uint64_t r = mix(seed + id * iters + i), r2 = mix(r), r3 = mix(r2);
    const int kind = (int)(r3 % 6);
    double a = operand(kind == 5 ? 1 : kind, r), b = operand(kind == 5 ? 1 : (r3 >> 8) % 5 == 0 ? 4 : kind, r2);
    double x = fabs(a);
    if (kind == 5) {
      // a next to q b for a 54-bit q: the quotient next to a representable number or a midpoint
      const double q = operand(1, r3), h = ldexp(1.0, ilogb(q) - 53);
      const double off = (r3 >> 60) & 1 ? 0.0 : h;
      a = fma(q, b, off * b);
      if ((r3 >> 61) & 1) a = as_double((uint64_t)__double_as_longlong(a) + ((r3 >> 62) & 1 ? 1 : -1));
      // x next to the square of a representable number or of a midpoint
      const double s = fabs(q);
      x = fma(s, s, 2.0 * s * off);
      if ((r3 >> 59) & 1) x = as_double((uint64_t)__double_as_longlong(x) + ((r3 >> 58) & 1 ? 1 : -1));
    }
    if (kind == 0 && (r3 >> 20) % 8 == 0) x = a;  // negative operands of the root
    if (!same(soft_div(a, b), __ddiv_rn(a, b))) {
      if (atomicAdd(bad, 1ull) == 0) {
        ex[0] = a;
        ex[1] = b;
      }
    }
    if (!same(soft_sqrt(x), __dsqrt_rn(x))) {
      if (atomicAdd(bad + 1, 1ull) == 0) ex[2] = x;
    }
    if (kind == 5) {  // factors of about 27 bits: products next to a tie
      a = as_double((uint64_t)__double_as_longlong(operand(1, r)) & ~0ull << (24 + (r3 >> 12) % 4));
      b = as_double((uint64_t)__double_as_longlong(operand(1, r2)) & ~0ull << (24 + (r3 >> 14) % 4));
      if ((r3 >> 57) & 1) b = as_double((uint64_t)__double_as_longlong(b) + 1);
    }
    if (!same(soft_mul(a, b), __dmul_rn(a, b))) {
      if (atomicAdd(bad + 2, 1ull) == 0) {
        ex[3] = a;
        ex[4] = b;
      }
    }
  }
}

int main() {
  unsigned long long* bad;
  double* ex;
  if (cudaMallocManaged(&bad, 24) != cudaSuccess || cudaMallocManaged(&ex, 40) != cudaSuccess) return 2;
  bad[0] = bad[1] = bad[2] = 0;
  for (int rep = 0; rep < 4; ++rep) check<<<1024, 256>>>(1234567ull + ((uint64_t)rep << 40), 256, bad, ex);
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    fprintf(stderr, "%s\n", cudaGetErrorString(e));
    return 2;
  }
  printf("268M operand pairs: %llu quotients, %llu roots and %llu products differ\n", bad[0], bad[1], bad[2]);
  if (bad[0]) fprintf(stderr, "division: %a / %a\n", ex[0], ex[1]);
  if (bad[1]) fprintf(stderr, "root: %a\n", ex[2]);
  if (bad[2]) fprintf(stderr, "product: %a * %a\n", ex[3], ex[4]);
  return bad[0] || bad[1] || bad[2] ? 1 : 0;
}
