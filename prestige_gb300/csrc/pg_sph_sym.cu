// The IEEE f64 step with each neighbour pair evaluated once (ARITH_F64_EXACT).
//
// The oracle's pair terms (oracle/prestige_oracle.hpp, sph_pair_loop) are, per particle i and
// neighbour j in walk order,
//   continuity  dr_i += m_j (w F),                  w = (v_i - v_j) . (x_i - x_j)
//   momentum    a_i  -= m_j (((P_i + P_j) + pi_ij) F) (x_i - x_j),
//               pi_ij = avk w / ((r^2 + eps h^2)(rho_i + rho_j)) where w < 0, else 0,
// with F, r^2 and w computed from the pair's differences.  In IEEE arithmetic every one of
// r^2, F, w, w F and X = ((P_i + P_j) + pi_ij) F is the same bit pattern from either side of
// the pair: negating both factors of a product is exact, the component sums run in the same
// order, and a + b == b + a.  Only m_j and the final difference vector belong to one side.  So
// the side with the lower slot evaluates the pair once and writes the symmetric value into both
// list entries; each particle then sums its own entries in list (walk) order, which is the
// oracle's order, bit for bit.
//
// Lists (sph_list_kernel) hold each slot's neighbours in ascending slot order: the entries below
// the slot's own index come first.  Per step:
//   sym_c1  for the entries above the slot (partner t > k): F, w, w F and r^2 + eps h^2 into the
//           slot's entry planes; t and the position of k in t's list (binary search: t's list is
//           ascending) into the mirror plane, and w F into t's entry there.
//   sym_c2  every entry in order: w F from the entry (own, or the mirror t wrote), times m_t,
//           into the continuity sum; then rho' and the packed {rho', P'} (the oracle's rho
//           update and Tait term).
//   sym_m1  for the entries above the slot: X from the stored F, w, r^2 + eps h^2 and the packed
//           {rho', P'} of both sides, into the slot's entry and through the mirror index.
//   sym_m2  every entry in order: X times m_t times the slot's own difference vector, into the
//           momentum sum; then the velocity and position update of fluid particles.
// A pair whose mirror entry does not exist (a list that reached its capacity before the partner:
// the partner's continued walk evaluates the pair itself) or was not written (the lower slot's
// list reached its capacity before this slot) is evaluated in full where it is read, and an
// overflowed list is followed by the rest of its candidate walk, evaluated in full, as in the
// other modes.
//
// The kernels are bound by the FP64 pipe and, beside it, by the latency of their loads.  Against FP64
// instructions for everything and all lanes of a warp at the same entry index (1M particles, ms: c1
// 4.6, c2 0.44, m1 1.56, m2 1.58): divisions and roots on the integer pipe 2.95 / 0.41 / 0.94 / 1.57;
// each lane from its own first entry above the slot, multiplications on the integer pipe and the
// loads pipelined 2.0 / 0.40 / 0.91 / 1.09 (FP64 pipe 64 / 34 / 35 / 71 % busy, issue slots 40 to 60 %);
// four threads per slot in c1 and m1 another 0.25 less together.
// Where a warp or two share a scheduler and latency decides, the FP64 multiplication is the faster
// one (two-sided passes at 6.5k particles: 0.118 ms a step against 0.153 with soft_mul; the dense DEM
// pass 0.296 against 0.368), so only these kernels use the integer one.  (Step of 1M moving
// particles 4.80 ms, with FP64 products 5.64; at rest on a regular lattice, where a zero factor in any lane
// takes the warp through both, 7.70 and 7.69; the 2D dam break of 6,518 70 us and 60.)
#include <cuda_runtime.h>
#include <stdint.h>

#include "pg_arith.cuh"
#include "pg_internal.cuh"
#include "pg_kernels.cuh"
#include "pg_sph_pass.cuh"

namespace pg {
namespace {

using namespace sphpass;

typedef OpsDI D;  // multiplications, divisions and roots on the integer pipe

// Entry planes of the per-entry store (a.fcache): doubles F, w, r^2 + eps h^2, S (w F after
// sym_c1, X after sym_m1), then a word with the mirror index and the partner (mirror_word), each plane
// in the tiled list layout.  S is indexed like the list; the others, which only the slot itself reads,
// by the number of the entry among those above the slot, so a warp whose lanes each start at their own
// first entry above the slot still reads and writes whole rows of them.
struct Planes {
  double* base;
  size_t plane;  // entries per plane
  __device__ __forceinline__ double* F(size_t e) const { return base + e; }
  __device__ __forceinline__ double* W(size_t e) const { return base + plane + e; }
  __device__ __forceinline__ double* R(size_t e) const { return base + 2 * plane + e; }
  __device__ __forceinline__ double* S(size_t e) const { return base + 3 * plane + e; }
  __device__ __forceinline__ uint32_t* M(size_t e) const { return (uint32_t*)(base + 4 * plane) + e; }
};

__device__ __forceinline__ Planes planes_of(const SphArgs& a) {
  Planes p;
  p.base = (double*)a.fcache;
  p.plane = (size_t)((a.n + kListTile - 1) / kListTile) * kListTile * a.cap;
  return p;
}

__device__ __forceinline__ size_t entry(uint32_t k, uint32_t q, uint32_t cap) {
  return list_base(k, cap) + (size_t)q * kListTile;
}

// The oracle's pair geometry and continuity factor from slot k's side: d = x_k - x_t, r^2, F, w.
template <int DIM>
__device__ __forceinline__ void pair_geometry(const SphC<double>& c, const double4_32a& Ai, const double4_32a& Bi,
                                              const double4_32a& Aj, const double4_32a& Bj, double* d, double& r2,
                                              double& F, double& w) {
  d[0] = D::sub(Ai.x, Aj.x);
  d[1] = D::sub(Ai.y, Aj.y);
  d[2] = DIM == 3 ? D::sub(Ai.z, Aj.z) : 0.0;
  r2 = D::add(D::mul(d[0], d[0]), D::mul(d[1], d[1]));
  if (DIM == 3) r2 = D::add(r2, D::mul(d[2], d[2]));
  const double r = D::sqrt(r2);
  const double q = D::mul(r, c.inv_h);
  const double tq = D::sub(2.0, q);
  const double Fnear = D::mul(c.fa, D::sub(D::mul(2.25, q), 3.0));
  const double Ffar = D::div(D::mul(c.fb, D::mul(tq, tq)), r);
  F = q < 1.0 ? Fnear : Ffar;
  const double dv0 = D::sub(Bi.x, Bj.x), dv1 = D::sub(Bi.y, Bj.y);
  const double dv2 = DIM == 3 ? D::sub(Bi.z, Bj.z) : 0.0;
  w = D::add(D::mul(dv0, d[0]), D::mul(dv1, d[1]));
  if (DIM == 3) w = D::add(w, D::mul(dv2, d[2]));
}

// X = ((P_k + P_t) + pi_kt) F, the oracle's operation order.
__device__ __forceinline__ double momentum_factor(const SphC<double>& c, double F, double w, double r2e,
                                                  const double2& qk, const double2& qt) {
  const double av = D::div(D::mul(c.avk, w), D::mul(r2e, D::add(qk.x, qt.x)));
  const double pij = w < 0.0 ? av : 0.0;
  return D::mul(D::add(D::add(qk.y, qt.y), pij), F);
}

// The oracle's neighbour test on the candidate walk (r^2 < 4h^2 and r^2 > 0).
template <int DIM>
__device__ __forceinline__ bool is_neighbor(const SphC<double>& c, const double4_32a& Ai, const double4_32a& Aj) {
  const double d0 = D::sub(Ai.x, Aj.x), d1 = D::sub(Ai.y, Aj.y);
  double r2 = D::add(D::mul(d0, d0), D::mul(d1, d1));
  if (DIM == 3) {
    const double d2 = D::sub(Ai.z, Aj.z);
    r2 = D::add(r2, D::mul(d2, d2));
  }
  return r2 < c.four_h2 && r2 > 0.0;
}

// The rest of the candidate walk of slot k after its list reached capacity, in walk order
// (rows z, then y; slots ascending), calling on_pair(t) for every neighbour.
template <int DIM, class OnPair>
__device__ __forceinline__ void resume_walk(const SphArgs& a, const SphK& K, uint32_t k, const double4_32a& Ai,
                                            OnPair&& on_pair) {
  const double4_32a* __restrict__ A = (const double4_32a*)a.s[0];
  continue_walk<DIM, false>(a, k, [&](uint32_t t) {
    if (is_neighbor<DIM>(K.d, Ai, A[t])) on_pair(t);
  });
}

// A pair without a stored value (a list at its capacity), everything from the packs; out of line, so the
// passes' common path does not hold its registers.
template <int DIM>
__device__ __noinline__ double full_wF(const SphC<double>* c, const double4_32a* A, const double4_32a* B, uint32_t k,
                                       uint32_t t) {
  double d[3], r2, F, w;
  pair_geometry<DIM>(*c, A[k], B[k], A[t], B[t], d, r2, F, w);
  return D::mul(w, F);
}
template <int DIM>
__device__ __noinline__ double full_X(const SphC<double>* c, const double4_32a* A, const double4_32a* B,
                                      const double2* Q, uint32_t k, uint32_t t) {
  double d[3], r2, F, w;
  pair_geometry<DIM>(*c, A[k], B[k], A[t], B[t], d, r2, F, w);
  return momentum_factor(*c, F, w, D::add(r2, c->eps_h2), Q[k], Q[t]);
}

// LANES threads share a slot in the pair-value kernels: thread `sub` takes every LANES-th entry (the values
// do not depend on who evaluates them).  With 8 slots to a warp the slots' entry counts differ less
// than with 32, and a small system fills more of the chip.
constexpr int kPairLanes = 4;

struct Slot {
  uint32_t k, id, L, sub;
  bool overflow;
};

template <int LANES = 1>
__device__ __forceinline__ bool slot_of(const SphArgs& a, Slot& s) {
  s.k = a.k_begin + lane_slot<LANES>(blockIdx.x, blockDim.x, threadIdx.x);
  s.sub = threadIdx.x % LANES;
  if (s.k >= a.k_end) return false;
  s.id = a.sorted_id[s.k];
  const uint32_t cnt = a.nlen[s.k];
  s.L = min(cnt, a.cap);
  s.overflow = cnt > a.cap;
  return true;
}

// split > 0: the lists of the slots from split on may still be being built (on another stream).
// A slot's pair values need its partners' complete lists, so the first launch (second == 0)
// takes the slots below split whose stored partners all lie below split (lists ascend, so the
// last stored entry decides) and the second launch, after all lists, the others.
template <int DIM>
__global__ void __launch_bounds__(kSphMaxThreads) sym_c1_kernel(SphArgs a, uint32_t split, int second) {
  chain_begin();
  Slot s;
  if (!slot_of<kPairLanes>(a, s)) return;
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  if (split) {
    const bool early = s.k < split && (s.L == 0 || my[(size_t)(s.L - 1) * kListTile] < split);
    if (early == (second != 0)) return;
  }
  const SphK& K = a.sys[sys_of_slot(a, s.id)];
  const double4_32a* __restrict__ A = (const double4_32a*)a.s[0];
  const double4_32a* __restrict__ B = (const double4_32a*)a.s[1];
  const Planes P = planes_of(a);
  const double4_32a Ai = A[s.k], Bi = B[s.k];
  // each lane from its own first entry above the slot: with all lanes at the same entry index a third
  // of them idled (21 of 32 active), while the FP64 pipe takes as long for 21 lanes as for 32
  const uint32_t q0 = lower_bound(my, s.L, s.k), U = s.L - q0;
  my += (size_t)q0 * kListTile;
  // the positions of k in the partners' lists first, kSearch searches at a time (each is a chain of
  // dependent loads)
  for (uint32_t j = s.sub; j < U; j += kPairLanes * kSearch) {
    uint32_t t[kSearch], m[kSearch];
#pragma unroll
    for (int i = 0; i < kSearch; ++i) t[i] = my[(size_t)min(j + i * kPairLanes, U - 1) * kListTile];
    find_in_lists(a, t, s.k, m);
#pragma unroll
    for (int i = 0; i < kSearch; ++i)
      if (j + i * kPairLanes < U) *P.M(entry(s.k, j + i * kPairLanes, a.cap)) = mirror_word(m[i], t[i], s.k);
  }
  if (s.sub >= U) return;
  // software pipeline: entries two ahead, the partner's records one ahead (each thread reads back the
  // entries it wrote above)
  constexpr uint32_t N = kPairLanes;
  const uint32_t last = s.sub + (U - 1 - s.sub) / N * N;  // the thread's last entry
  Mirror m = mirror_of(*P.M(entry(s.k, s.sub, a.cap)), s.k, my, s.sub);
  uint32_t next = *P.M(entry(s.k, min(s.sub + N, last), a.cap));
  double4_32a Aj = A[m.slot], Bj = B[m.slot];
  for (uint32_t j = s.sub; j < U; j += N) {
    const uint32_t next2 = *P.M(entry(s.k, min(j + 2 * N, last), a.cap));
    const Mirror mn = mirror_of(next, s.k, my, min(j + N, last));
    const double4_32a An = A[mn.slot], Bn = B[mn.slot];
    double d[3], r2, F, w;
    pair_geometry<DIM>(K.d, Ai, Bi, Aj, Bj, d, r2, F, w);
    const double wF = D::mul(w, F);
    const size_t e = entry(s.k, j, a.cap);
    *P.F(e) = F;
    *P.W(e) = w;
    *P.R(e) = D::add(r2, K.d.eps_h2);
    *P.S(entry(s.k, q0 + j, a.cap)) = wF;
    if (m.pos != kNoPos) *P.S(entry(m.slot, m.pos, a.cap)) = wF;
    m = mn;
    next = next2;
    Aj = An;
    Bj = Bn;
  }
}

template <int DIM>
__global__ void __launch_bounds__(kSphMaxThreads) sym_c2_kernel(SphArgs a) {
  chain_begin();
  Slot s;
  if (!slot_of(a, s)) return;
  const SphK& K = a.sys[sys_of_slot(a, s.id)];
  const SphC<double>& c = K.d;
  const double4_32a* __restrict__ A = (const double4_32a*)a.s[0];
  const double4_32a* __restrict__ B = (const double4_32a*)a.s[1];
  const Planes P = planes_of(a);
  const double4_32a Ai = A[s.k];
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  auto full = [&](uint32_t t) { return full_wF<DIM>(&c, A, B, s.k, t); };
  // software pipeline: list entries two ahead, the partner's mass and list length and the
  // entry's stored value one ahead (the pass waits on these loads; its FP64 work is two
  // operations per entry, summed in list order)
  double dr = 0.0;
  const uint32_t L = s.L;
  uint32_t t = L > 0 ? my[0] : 0u;
  uint32_t tn = L > 1 ? my[kListTile] : 0u;
  double mt = L > 0 ? A[t].w : 0.0;
  uint32_t nl = L > 0 ? a.nlen[t] : 0u;
  double sv = L > 0 ? *P.S(entry(s.k, 0, a.cap)) : 0.0;
  for (uint32_t q = 0; q < L; ++q) {
    if (q + kL2Ahead < L) {
      prefetch_l2(my + (size_t)(q + kL2Ahead) * kListTile);
      prefetch_l2(P.S(entry(s.k, q + kL2Ahead, a.cap)));
    }
    const uint32_t tnn = q + 2 < L ? my[(size_t)(q + 2) * kListTile] : 0u;
    const double mtn = q + 1 < L ? A[tn].w : 0.0;
    const uint32_t nln = q + 1 < L ? a.nlen[tn] : 0u;
    const double svn = q + 1 < L ? *P.S(entry(s.k, q + 1, a.cap)) : 0.0;
    // the value is in the entry unless the partner below is one whose list reached its capacity before
    // this slot (lists ascend: then its last stored entry is below the slot)
    const bool stored = t > s.k || nl <= a.cap || a.nlist[entry(t, a.cap - 1, a.cap)] >= s.k;
    dr = D::add(dr, D::mul(mt, stored ? sv : full(t)));
    t = tn;
    tn = tnn;
    mt = mtn;
    nl = nln;
    sv = svn;
  }
  if (s.overflow) resume_walk<DIM>(a, K, s.k, Ai, [&](uint32_t t) { dr = D::add(dr, D::mul(A[t].w, full(t))); });
  double* rho = (double*)a.rho;
  const double rn = D::add(rho[s.id], D::mul(c.dt, dr));
  rho[s.id] = rn;
  ((double2*)a.s[2])[s.k] = make_double2(rn, tait_pterm<OpsD>(c, K.gamma, rn));
}

template <int DIM>
__global__ void __launch_bounds__(kSphMaxThreads) sym_m1_kernel(SphArgs a) {
  chain_begin();
  Slot s;
  if (!slot_of<kPairLanes>(a, s)) return;
  const SphK& K = a.sys[sys_of_slot(a, s.id)];
  const double2* __restrict__ Q = (const double2*)a.s[2];
  const Planes P = planes_of(a);
  const double2 qk = Q[s.k];
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  // each lane from its own first entry above the slot, as in sym_c1; the pass waits on its loads, so
  // the partner's index is loaded two entries ahead and everything else one ahead
  const uint32_t q0 = lower_bound(my, s.L, s.k), U = s.L - q0;
  if (s.sub >= U) return;
  my += (size_t)q0 * kListTile;
  constexpr uint32_t N = kPairLanes;
  Mirror m = mirror_of(*P.M(entry(s.k, s.sub, a.cap)), s.k, my, s.sub);
  uint32_t next = *P.M(entry(s.k, min(s.sub + N, U - 1), a.cap));
  size_t e = entry(s.k, s.sub, a.cap);
  double F = *P.F(e), w = *P.W(e), r2e = *P.R(e);
  double2 qt = Q[m.slot];
  for (uint32_t j = s.sub; j < U; j += N) {
    const uint32_t next2 = *P.M(entry(s.k, min(j + 2 * N, U - 1), a.cap));
    const Mirror mn = mirror_of(next, s.k, my, min(j + N, U - 1));
    e = entry(s.k, min(j + N, U - 1), a.cap);
    const double Fn = *P.F(e), wn = *P.W(e), rn = *P.R(e);
    const double2 qn = Q[mn.slot];
    const double X = momentum_factor(K.d, F, w, r2e, qk, qt);
    *P.S(entry(s.k, q0 + j, a.cap)) = X;
    if (m.pos != kNoPos) *P.S(entry(m.slot, m.pos, a.cap)) = X;
    m = mn;
    next = next2;
    F = Fn;
    w = wn;
    r2e = rn;
    qt = qn;
  }
}

template <int DIM>
__global__ void __launch_bounds__(kSphMaxThreads) sym_m2_kernel(SphArgs a) {
  chain_begin();
  Slot s;
  if (!slot_of(a, s)) return;
  const SphK& K = a.sys[sys_of_slot(a, s.id)];
  const SphC<double>& c = K.d;
  const double4_32a* __restrict__ A = (const double4_32a*)a.s[0];
  const double4_32a* __restrict__ B = (const double4_32a*)a.s[1];
  const double2* __restrict__ Q = (const double2*)a.s[2];
  const Planes P = planes_of(a);
  const double4_32a Ai = A[s.k];
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  double acc[3] = {0.0, 0.0, 0.0};
  auto full = [&](uint32_t t) { return full_X<DIM>(&c, A, B, Q, s.k, t); };
  auto add = [&](const double4_32a& Aj, double X) {
    const double coef = D::mul(Aj.w, X);
    acc[0] = D::sub(acc[0], D::mul(coef, D::sub(Ai.x, Aj.x)));
    acc[1] = D::sub(acc[1], D::mul(coef, D::sub(Ai.y, Aj.y)));
    if (DIM == 3) acc[2] = D::sub(acc[2], D::mul(coef, D::sub(Ai.z, Aj.z)));
  };
  // software pipeline: list entries two ahead; the partner's record and list length and the entry's
  // stored value one ahead
  const uint32_t L = s.L;
  if (L > 0) {
    uint32_t t = my[0], tn = my[(size_t)min(1u, L - 1) * kListTile];
    double4_32a Aj = A[t];
    uint32_t nl = a.nlen[t];
    double X = *P.S(entry(s.k, 0, a.cap));
    for (uint32_t q = 0; q < L; ++q) {
      const uint32_t tnn = my[(size_t)min(q + 2, L - 1) * kListTile];
      const double4_32a An = A[tn];
      const uint32_t nln = a.nlen[tn];
      const double Xn = *P.S(entry(s.k, min(q + 1, L - 1), a.cap));
      const bool stored = t > s.k || nl <= a.cap || a.nlist[entry(t, a.cap - 1, a.cap)] >= s.k;  // as in sym_c2
      add(Aj, stored ? X : full(t));
      t = tn;
      tn = tnn;
      Aj = An;
      nl = nln;
      X = Xn;
    }
  }
  if (s.overflow) resume_walk<DIM>(a, K, s.k, Ai, [&](uint32_t t) { add(A[t], full(t)); });
  if (s.id < K.fluid_end) {
    double* pos = (double*)a.pos;
    double* vel = (double*)a.vel;
#pragma unroll
    for (int cc = 0; cc < DIM; ++cc) {
      const size_t o = (size_t)s.id * DIM + cc;
      const double v = D::add(vel[o], D::mul(c.dt, D::add(acc[cc], c.g[cc])));
      vel[o] = v;
      pos[o] = D::add(pos[o], D::mul(c.dt, v));
    }
  }
}

typedef void (*SymKernel)(SphArgs);

template <int DIM>
SymKernel sym_kernel(int part) {
  switch (part) {
    case 1: return sym_c2_kernel<DIM>;
    case 2: return sym_m1_kernel<DIM>;
    case 3: return sym_m2_kernel<DIM>;
    default: return nullptr;
  }
}

}  // namespace

size_t sph_sym_entry_bytes() { return 4 * sizeof(double) + sizeof(uint32_t); }

int launch_sph_sym(cudaStream_t st, const SphArgs& a, int part, int block, uint32_t split, int second) {
  SymKernel kern = a.dim == 2 ? sym_kernel<2>(part) : sym_kernel<3>(part);
  if (!kern && part != 0) {
    set_error("unknown part %d of the pair-once step", part);
    return PG_EINVAL;
  }
  if (block < 32 || block > kSphMaxThreads || block % 32) {
    set_error("block size %d must be a multiple of 32 in 32..%d", block, kSphMaxThreads);
    return PG_EINVAL;
  }
  if (a.k_end <= a.k_begin) return PG_OK;
  const int lanes = part == 0 || part == 2 ? kPairLanes : 1;
  const unsigned blocks = (unsigned)(((size_t)(a.k_end - a.k_begin) * lanes + block - 1) / block);
  if (part == 0) {
    PG_CUDA_TRY(launch_chained(st, a.chained != 0, a.dim == 2 ? sym_c1_kernel<2> : sym_c1_kernel<3>, blocks,
                               (unsigned)block, a, split, second));
  } else {
    PG_CUDA_TRY(launch_chained(st, a.chained != 0, kern, blocks, (unsigned)block, a));
  }
  return PG_OK;
}

}  // namespace pg
