// The FP64 adjoint passes with each neighbour pair evaluated once (IEEE f64 handles).
//
// The adjoint of one step (pg_adjoint.cu) sums, for particle i over its neighbours j, the
// derivatives of the pair terms Lam_M and Lam_C.  With x = x_i - x_j, v = v_i - v_j and
// E = m_j abar_i - m_i abar_j, particle i's share of a pair is
//   momentum     gx_i += a1 x + b1 v - F S E,   gv_i += b1 x,   gr_i -= F (x.E) (P'_i - Pi / rho_ij)
//   continuity   gx_i += G w D x + F D v,       gv_i += F D x
// where a1, b1, F, G, S, Pi, w, x.E and D are the same from either side of the pair while x, v
// and E change sign.  So j's share is the negated vector of i's (and its own P'_j in gr), and
// the lower slot of a pair evaluates it once:
//   adj_mirror  for each entry above the slot, the slot's position in the partner's list
//           (binary search: the partner's list is ascending), or none.
//   adj_a1  (entries above the slot) the momentum terms; its own share into per-slot partial
//           sums; the partner's share (the vectors, F x.E and Pi / rho_ij) into the partner's list
//           entry at the mirror index; the pair's continuity vectors U1 = G w x + F v and
//           U2 = F x and the partner's mass into the slot's own entry; the parameter derivatives
//           of the pair whole (half of each when the partner evaluates its side itself).
//   adj_a2  (entries below the slot, in list order) the partners' shares, then the momentum
//           update of lx, lv, lr, the parameter sums and dbar = dt lr for the continuity pass.
//   adj_c1 / adj_c2  the same for the continuity terms: the slot's share is D U1 and D U2 with
//           D = dbar_k m_t + dbar_t m_k (dbar from adj_a2), the partner's the negated vectors.
// A pair that is not held by both lists (a list that reached its capacity) is evaluated by each
// side for itself, as in the two-sided passes, with half of the parameter derivatives each; the
// rest of an overflowed list's walk likewise.  The sums run in a different order from the
// two-sided passes, within the adjoint's tolerance against the dual-number oracle.
#include <cuda_runtime.h>
#include <stdint.h>

#include "pg_arith.cuh"
#include "pg_internal.cuh"
#include "pg_kernels.cuh"
#include "pg_sph_pass.cuh"

namespace pg {
namespace {

using namespace sphpass;

constexpr int kPlanes = 15;  // doubles per list entry (plus the word with mirror index and partner)
// the partner's momentum share (Vx, Vv, F x.E, Pi / rho_ij); for the continuity pass, the pair's
// vectors U1 = G w x + F v and U2 = F x and the partner's mass (own entries above the slot).  The first
// group is indexed like the list; the second and the mirror words (mirror_word), which only the slot
// itself reads, by the number of the entry among those above the slot, so lanes that each start at
// their own first entry above the slot read and write whole rows of them.
enum { kMx = 0, kMv = 3, kFxE = 6, kPIrb = 7, kU1 = 8, kU2 = 11, kMt = 14 };
constexpr int kAdjBlock = 128;
constexpr int kAdjLanes = 4;  // threads per slot
constexpr int kSlotSums = 9;  // per-slot partial sums: gx (3), gv (3), gr, gal, gB

struct Planes {
  double* base;
  size_t plane;  // entries per plane
  __device__ __forceinline__ double& at(int j, size_t e) const { return base[j * plane + e]; }
  __device__ __forceinline__ uint32_t& mirror(size_t e) const { return ((uint32_t*)(base + kPlanes * plane))[e]; }
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

// Slot t's list holds slot k (a neighbour above t) as a stored entry.
__device__ __forceinline__ bool holds(const SphArgs& a, uint32_t t, uint32_t k) {
  if (a.nlen[t] <= a.cap) return true;
  return a.nlist[entry(t, a.cap - 1, a.cap)] >= k;
}

// The slot-ordered packs of the adjoint step (adjoint_prep_kernel):
//   s0 X {x, y, z, m}  s1 V {v, rho'}  s2 Q {P, P', P/B}  s3 A {abar}  s5 dbar  pf FP32 x
//   s6 per-slot partial sums (kSlotSums planes of n doubles)
struct Packs {
  const double4_32a *X, *V, *Q, *A;
  const double* DB;
  double* PS;
  __device__ __forceinline__ Packs(const SphArgs& a)
      : X((const double4_32a*)a.s[0]), V((const double4_32a*)a.s[1]), Q((const double4_32a*)a.s[2]),
        A((const double4_32a*)a.s[3]), DB((const double*)a.s[5]), PS((double*)a.s[6]) {}
};

// Pair geometry from slot k's side: x, v, r^2, F = (dW/dr)/r, G = (dF/dr)/r, w = v . x.
template <int DIM>
struct Geo {
  double d[3], dv[3], r2, F, G, w;
};

template <int DIM>
__device__ __forceinline__ Geo<DIM> geometry(const SphC<double>& c, const double4_32a& xk, const double4_32a& vk,
                                             const double4_32a& xt, const double4_32a& vt) {
  Geo<DIM> g;
  g.d[0] = xk.x - xt.x;
  g.d[1] = xk.y - xt.y;
  g.d[2] = DIM == 3 ? xk.z - xt.z : 0.0;
  g.r2 = __dadd_rn(__dmul_rn(g.d[0], g.d[0]), __dmul_rn(g.d[1], g.d[1]));
  if (DIM == 3) g.r2 = __dadd_rn(g.r2, __dmul_rn(g.d[2], g.d[2]));
  const double inv_r = soft_div(1.0, soft_sqrt(g.r2));  // off the FP64 pipe (pg_softf64.cuh)
  const double r = g.r2 * inv_r;
  const double q = r * c.inv_h;
  if (q < 1.0) {
    g.F = c.fa * (2.25 * q - 3.0);
    g.G = c.fa * 2.25 * c.inv_h * inv_r;
  } else {
    const double tq = 2.0 - q;
    g.F = c.fb * tq * tq * inv_r;
    g.G = -(c.fb * tq * inv_r) * (2.0 * c.inv_h + tq * inv_r) * inv_r;
  }
  g.dv[0] = vk.x - vt.x;
  g.dv[1] = vk.y - vt.y;
  g.dv[2] = DIM == 3 ? vk.z - vt.z : 0.0;
  g.w = g.dv[0] * g.d[0] + g.dv[1] * g.d[1];
  if (DIM == 3) g.w += g.dv[2] * g.d[2];
  return g;
}

// The oracle's neighbour test (r^2 < 4h^2 and r^2 > 0), for the continued walks.
template <int DIM>
__device__ __forceinline__ bool is_neighbor(const SphC<double>& c, const double4_32a& xk, const double4_32a& xt) {
  const double d0 = xk.x - xt.x, d1 = xk.y - xt.y;
  double r2 = __dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1));
  if (DIM == 3) {
    const double d2 = xk.z - xt.z;
    r2 = __dadd_rn(r2, __dmul_rn(d2, d2));
  }
  return r2 < c.four_h2 && r2 > 0.0;
}

// The momentum-adjoint terms of pair (k, t) from k's side.
template <int DIM>
struct MomTerms {
  double Vx[3], Vv[3], FxE, PIrb, gal, gB;  // gal, gB: the whole pair's parameter derivatives
  double U1[3], U2[3], mt;                  // the continuity share is D U1, D U2
};

template <int DIM>
__device__ __forceinline__ MomTerms<DIM> mom_terms(const SphK& K, const Packs& P, uint32_t k, uint32_t t,
                                                   const double4_32a& xk, const double4_32a& vk) {
  const SphC<double>& c = K.d;
  const double4_32a xt = P.X[t], vt = P.V[t], qk = P.Q[k], qt = P.Q[t], ak = P.A[k], at = P.A[t];
  const Geo<DIM> g = geometry<DIM>(c, xk, vk, xt, vt);
  const double mk = xk.w, mt = xt.w;
  const double rb = vk.w + vt.w;
  const double e = g.r2 + c.eps_h2;
  // one reciprocal serves the four quotients of the terms
  const double inv_erb = soft_div(1.0, e * rb);
  const double inv_e = rb * inv_erb, inv_rb = e * inv_erb;
  double c1 = 0.0, c1a = 0.0;
  if (g.w < 0.0) {
    const double base = inv_e * inv_rb;
    c1 = c.avk * base;
    c1a = K.avk_alpha * base;
  }
  const double PI = c1 * g.w;
  const double S = qk.x + qt.x + PI;
  const double E[3] = {mt * ak.x - mk * at.x, mt * ak.y - mk * at.y, DIM == 3 ? mt * ak.z - mk * at.z : 0.0};
  double xE = 0.0;
#pragma unroll
  for (int cc = 0; cc < DIM; ++cc) xE += g.d[cc] * E[cc];
  const double a1 = -g.G * S * xE + 2.0 * g.F * xE * PI * inv_e;
  const double b1 = -g.F * c1 * xE;
  const double fs = g.F * S;
  MomTerms<DIM> m;
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    m.Vx[cc] = cc < DIM ? a1 * g.d[cc] + b1 * g.dv[cc] - fs * E[cc] : 0.0;
    m.Vv[cc] = cc < DIM ? b1 * g.d[cc] : 0.0;
  }
  m.FxE = g.F * xE;
  m.PIrb = PI * inv_rb;
  m.gal = m.FxE * c1a * g.w;
  m.gB = m.FxE * (qk.z + qt.z);
  const double GW = g.G * g.w;
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    m.U1[cc] = cc < DIM ? GW * g.d[cc] + g.F * g.dv[cc] : 0.0;
    m.U2[cc] = cc < DIM ? g.F * g.d[cc] : 0.0;
  }
  m.mt = mt;
  return m;
}

struct Sums {
  double gx[3], gv[3], gr, gal, gB;
};

template <int DIM>
__device__ __forceinline__ void add_own(Sums& s, const MomTerms<DIM>& m, double Pdk, double share) {
#pragma unroll
  for (int cc = 0; cc < DIM; ++cc) {
    s.gx[cc] += m.Vx[cc];
    s.gv[cc] += m.Vv[cc];
  }
  s.gr -= m.FxE * (Pdk - m.PIrb);
  s.gal -= share * m.gal;
  s.gB -= share * m.gB;
}

// The rest of the candidate walk of slot k after its list reached capacity (walk order).
template <int DIM, class OnPair>
__device__ __forceinline__ void resume_walk(const SphArgs& a, const SphK& K, const Packs& P, uint32_t k,
                                            const double4_32a& xk, OnPair&& on_pair) {
  continue_walk<DIM, false>(a, k, [&](uint32_t t) {
    if (is_neighbor<DIM>(K.d, xk, P.X[t])) on_pair(t);
  });
}

// LANES threads share a slot: thread `sub` takes every LANES-th entry of its loops and the
// partial sums are added at the end in a fixed order.
template <int LANES>
struct Slot {
  uint32_t k, id, L, sub;
  bool overflow;
};

template <int LANES>
__device__ __forceinline__ bool slot_of(const SphArgs& a, Slot<LANES>& s) {
  s.k = lane_slot<LANES>(blockIdx.x, blockDim.x, threadIdx.x);
  s.sub = threadIdx.x % LANES;
  if (s.k >= a.n) return false;
  s.id = a.sorted_id[s.k];
  const uint32_t cnt = a.nlen[s.k];
  s.L = min(cnt, a.cap);
  s.overflow = cnt > a.cap;
  return true;
}

// v summed over the threads of the slot (all of them call this; every one gets the sum).
template <int LANES>
__device__ __forceinline__ double lane_sum(double v) {
  if (LANES == 1) return v;
  const int lane = threadIdx.x & 31;
  const unsigned group = ((1u << LANES) - 1u) << (lane & ~(LANES - 1));
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) v += __shfl_xor_sync(group, v, o);
  return v;
}

template <int LANES>
__device__ __forceinline__ void lane_sums(Sums& s, int count) {
  if (LANES == 1) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    s.gx[c] = lane_sum<LANES>(s.gx[c]);
    s.gv[c] = lane_sum<LANES>(s.gv[c]);
  }
  if (count > 6) {
    s.gr = lane_sum<LANES>(s.gr);
    s.gal = lane_sum<LANES>(s.gal);
    s.gB = lane_sum<LANES>(s.gB);
  }
}

__device__ __forceinline__ void store_sums(const SphArgs& a, const Packs& P, uint32_t k, const Sums& s, int count) {
  const double v[kSlotSums] = {s.gx[0], s.gx[1], s.gx[2], s.gv[0], s.gv[1], s.gv[2], s.gr, s.gal, s.gB};
  for (int j = 0; j < count; ++j) P.PS[(size_t)j * a.n + k] = v[j];
}

__device__ __forceinline__ void add_stored_sums(const SphArgs& a, const Packs& P, uint32_t k, Sums& s, int count) {
  double v[kSlotSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int j = 0; j < count; ++j) v[j] = P.PS[(size_t)j * a.n + k];
  for (int c = 0; c < 3; ++c) {
    s.gx[c] += v[c];
    s.gv[c] += v[3 + c];
  }
  s.gr += v[6];
  s.gal += v[7];
  s.gB += v[8];
}

// The mirror index of every entry above its slot: the position of the slot in the partner's
// list (a binary search, latency-bound; apart from the FP64 work of adj_a1 it runs at full
// occupancy).
template <int LANES>
__global__ void __launch_bounds__(kSphMaxThreads) adj_mirror_kernel(SphArgs a) {
  chain_begin();
  Slot<LANES> s;
  if (!slot_of(a, s)) return;
  const Planes E = planes_of(a);
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  const uint32_t q0 = lower_bound(my, s.L, s.k), U = s.L - q0;
  my += (size_t)q0 * kListTile;
  for (uint32_t j = s.sub * kSearch; j < U; j += LANES * kSearch) {
    uint32_t t[kSearch], m[kSearch];
#pragma unroll
    for (int i = 0; i < kSearch; ++i) t[i] = my[(size_t)min(j + i, U - 1) * kListTile];
    find_in_lists(a, t, s.k, m);
#pragma unroll
    for (int i = 0; i < kSearch; ++i)
      if (j + i < U) E.mirror(entry(s.k, j + i, a.cap)) = mirror_word(m[i], t[i], s.k);
  }
}

template <int DIM, int LANES>
__global__ void __launch_bounds__(kSphMaxThreads) adj_a1_kernel(SphArgs a) {
  chain_begin();
  Slot<LANES> s;
  if (!slot_of(a, s)) return;
  const SphK& K = a.sys[0];
  const Packs P(a);
  const Planes E = planes_of(a);
  const double4_32a xk = P.X[s.k], vk = P.V[s.k];
  const double Pdk = P.Q[s.k].y;
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  Sums sum = {{0, 0, 0}, {0, 0, 0}, 0, 0, 0};
  // each lane from its own first entry above the slot, so the lanes of a warp evaluate their
  // pairs in the same iterations
  const uint32_t q0 = lower_bound(my, s.L, s.k), U = s.L - q0;
  my += (size_t)q0 * kListTile;
  for (uint32_t j = s.sub; j < U; j += LANES) {
    const size_t e = entry(s.k, j, a.cap);
    const Mirror mt = mirror_of(E.mirror(e), s.k, my, j);
    const MomTerms<DIM> m = mom_terms<DIM>(K, P, s.k, mt.slot, xk, vk);
#pragma unroll
    for (int cc = 0; cc < DIM; ++cc) {
      E.at(kU1 + cc, e) = m.U1[cc];
      E.at(kU2 + cc, e) = m.U2[cc];
    }
    E.at(kMt, e) = m.mt;
    if (mt.pos != kNoPos) {
      const size_t f = entry(mt.slot, mt.pos, a.cap);
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        E.at(kMx + cc, f) = m.Vx[cc];
        E.at(kMv + cc, f) = m.Vv[cc];
      }
      E.at(kFxE, f) = m.FxE;
      E.at(kPIrb, f) = m.PIrb;
    }
    add_own<DIM>(sum, m, Pdk, mt.pos != kNoPos ? 1.0 : 0.5);
  }
  lane_sums<LANES>(sum, kSlotSums);
  if (s.sub == 0) store_sums(a, P, s.k, sum, kSlotSums);
}

template <int DIM, int LANES>
__global__ void __launch_bounds__(kSphMaxThreads) adj_a2_kernel(SphArgs a) {
  chain_begin();
  Slot<LANES> s;
  if (!slot_of(a, s)) return;
  const SphK& K = a.sys[0];
  const Packs P(a);
  const Planes E = planes_of(a);
  const double4_32a xk = P.X[s.k], vk = P.V[s.k];
  const double Pdk = P.Q[s.k].y;
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  Sums sum = {{0, 0, 0}, {0, 0, 0}, 0, 0, 0};
  const uint32_t below = lower_bound(my, s.L, s.k);  // the entries below the slot come first
  for (uint32_t q = s.sub; q < below; q += LANES) {
    const uint32_t t = my[(size_t)q * kListTile];
    if (holds(a, t, s.k)) {  // t's share of the pair was written here by t: negate it
      const size_t e = entry(s.k, q, a.cap);
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        sum.gx[cc] -= E.at(kMx + cc, e);
        sum.gv[cc] -= E.at(kMv + cc, e);
      }
      sum.gr -= E.at(kFxE, e) * (Pdk - E.at(kPIrb, e));
    } else {
      add_own<DIM>(sum, mom_terms<DIM>(K, P, s.k, t, xk, vk), Pdk, 0.5);
    }
  }
  if (s.overflow && s.sub == 0)
    resume_walk<DIM>(a, K, P, s.k, xk,
                     [&](uint32_t t) { add_own<DIM>(sum, mom_terms<DIM>(K, P, s.k, t, xk, vk), Pdk, 0.5); });
  lane_sums<LANES>(sum, kSlotSums);
  if (s.sub != 0) return;
  add_stored_sums(a, P, s.k, sum, kSlotSums);
  // the momentum adjoint's update: lx += gx, lv += dt lx' (fluid) + gv, lr += gr, dbar = dt lr for
  // the continuity pass, and the parameter sums
  double* lx = (double*)a.lam[0];
  double* lv = (double*)a.lam[1];
  double* lr = (double*)a.lam[2];
  const bool fluid = s.id < K.fluid_end;
  const double dt = K.d.dt;
#pragma unroll
  for (int cc = 0; cc < DIM; ++cc) {
    const size_t o = (size_t)s.id * DIM + cc;
    const double lxo = lx[o];
    lx[o] = lxo + sum.gx[cc];
    lv[o] = (fluid ? lv[o] + dt * lxo : lv[o]) + sum.gv[cc];
  }
  const double lrt = lr[s.id] + sum.gr;
  lr[s.id] = lrt;
  ((double*)a.s[5])[s.k] = dt * lrt;
  ((double*)a.lam[3])[s.id] += sum.gal;
  ((double*)a.lam[4])[s.id] += sum.gB;
}

// The continuity-adjoint share of a pair from the slot's side is D U1 and D U2, with
// D = dbar_k m_t + dbar_t m_k, U1 = G w x + F v and U2 = F x.
template <int DIM>
__device__ __forceinline__ void cont_full(const SphK& K, const Packs& P, uint32_t k, uint32_t t, const double4_32a& xk,
                                          const double4_32a& vk, Sums& sum) {
  const double4_32a xt = P.X[t];
  const Geo<DIM> g = geometry<DIM>(K.d, xk, vk, xt, P.V[t]);
  const double D = P.DB[k] * xt.w + P.DB[t] * xk.w;
  const double GW = g.G * g.w;
#pragma unroll
  for (int cc = 0; cc < DIM; ++cc) {
    sum.gx[cc] += D * (GW * g.d[cc] + g.F * g.dv[cc]);
    sum.gv[cc] += D * (g.F * g.d[cc]);
  }
}

template <int DIM, int LANES>
__global__ void __launch_bounds__(kSphMaxThreads) adj_c1_kernel(SphArgs a) {
  chain_begin();
  Slot<LANES> s;
  if (!slot_of(a, s)) return;
  const Packs P(a);
  const Planes E = planes_of(a);
  const double mk = P.X[s.k].w, dbk = P.DB[s.k];
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  Sums sum = {{0, 0, 0}, {0, 0, 0}, 0, 0, 0};
  // this pass waits on its loads: the partner two entries ahead, everything else one ahead
  const uint32_t q0 = lower_bound(my, s.L, s.k), U = s.L - q0;
  my += (size_t)q0 * kListTile;
  if (s.sub < U) {
    auto row = [&](uint32_t j) { return entry(s.k, min(j, U - 1), a.cap); };
    struct Vals {
      double u1[DIM], u2[DIM], mt, db;
    };
    auto load = [&](size_t e, uint32_t t, Vals& v) {
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        v.u1[cc] = E.at(kU1 + cc, e);
        v.u2[cc] = E.at(kU2 + cc, e);
      }
      v.mt = E.at(kMt, e);
      v.db = P.DB[t];
    };
    Mirror m = mirror_of(E.mirror(row(s.sub)), s.k, my, s.sub);
    uint32_t next = E.mirror(row(s.sub + LANES));
    Vals v, vn;
    load(row(s.sub), m.slot, v);
    for (uint32_t j = s.sub; j < U; j += LANES) {
      const uint32_t next2 = E.mirror(row(j + 2 * LANES));
      const Mirror mn = mirror_of(next, s.k, my, min(j + LANES, U - 1));
      load(row(j + LANES), mn.slot, vn);
      const double D = dbk * v.mt + v.db * mk;
      double Vx[DIM], Vv[DIM];
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        Vx[cc] = D * v.u1[cc];
        Vv[cc] = D * v.u2[cc];
        sum.gx[cc] += Vx[cc];
        sum.gv[cc] += Vv[cc];
      }
      if (m.pos != kNoPos) {
        const size_t f = entry(m.slot, m.pos, a.cap);
#pragma unroll
        for (int cc = 0; cc < DIM; ++cc) {
          E.at(kMx + cc, f) = Vx[cc];
          E.at(kMv + cc, f) = Vv[cc];
        }
      }
      m = mn;
      next = next2;
      v = vn;
    }
  }
  lane_sums<LANES>(sum, 6);
  if (s.sub == 0) store_sums(a, P, s.k, sum, 6);
}

template <int DIM, int LANES>
__global__ void __launch_bounds__(kSphMaxThreads) adj_c2_kernel(SphArgs a) {
  chain_begin();
  Slot<LANES> s;
  if (!slot_of(a, s)) return;
  const SphK& K = a.sys[0];
  const Packs P(a);
  const Planes E = planes_of(a);
  const double4_32a xk = P.X[s.k], vk = P.V[s.k];
  const uint32_t* __restrict__ my = a.nlist + list_base(s.k, a.cap);
  Sums sum = {{0, 0, 0}, {0, 0, 0}, 0, 0, 0};
  const uint32_t below = lower_bound(my, s.L, s.k);
  for (uint32_t q = s.sub; q < below; q += LANES) {
    const uint32_t t = my[(size_t)q * kListTile];
    if (holds(a, t, s.k)) {
      const size_t e = entry(s.k, q, a.cap);
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        sum.gx[cc] -= E.at(kMx + cc, e);
        sum.gv[cc] -= E.at(kMv + cc, e);
      }
    } else {
      cont_full<DIM>(K, P, s.k, t, xk, vk, sum);
    }
  }
  if (s.overflow && s.sub == 0)
    resume_walk<DIM>(a, K, P, s.k, xk, [&](uint32_t t) { cont_full<DIM>(K, P, s.k, t, xk, vk, sum); });
  lane_sums<LANES>(sum, 6);
  if (s.sub != 0) return;
  add_stored_sums(a, P, s.k, sum, 6);
  double* lx = (double*)a.lam[0];
  double* lv = (double*)a.lam[1];
#pragma unroll
  for (int cc = 0; cc < DIM; ++cc) {
    const size_t o = (size_t)s.id * DIM + cc;
    lx[o] += sum.gx[cc];
    lv[o] += sum.gv[cc];
  }
}

typedef void (*AdjSymKernel)(SphArgs);

template <int DIM, int LANES>
AdjSymKernel adj_sym_kernel(int part) {
  switch (part) {
    case 0: return adj_mirror_kernel<LANES>;
    case 1: return adj_a1_kernel<DIM, LANES>;
    case 2: return adj_a2_kernel<DIM, LANES>;
    case 3: return adj_c1_kernel<DIM, LANES>;
    case 4: return adj_c2_kernel<DIM, LANES>;
    default: return nullptr;
  }
}

}  // namespace

size_t adjoint_sym_entry_bytes() { return kPlanes * sizeof(double) + sizeof(uint32_t); }
size_t adjoint_sym_slot_bytes() { return kSlotSums * sizeof(double); }

int launch_adjoint_sym(cudaStream_t st, const SphArgs& a, int part) {
  AdjSymKernel kern = a.dim == 2 ? adj_sym_kernel<2, kAdjLanes>(part) : adj_sym_kernel<3, kAdjLanes>(part);
  if (!kern) {
    set_error("unknown part %d of the pair-once adjoint", part);
    return PG_EINVAL;
  }
  if (a.n == 0) return PG_OK;
  const unsigned blocks = (unsigned)(((size_t)a.n * kAdjLanes + kAdjBlock - 1) / kAdjBlock);
  PG_CUDA_TRY(launch_chained(st, a.chained != 0, kern, blocks, kAdjBlock, a));
  return PG_OK;
}

}  // namespace pg
