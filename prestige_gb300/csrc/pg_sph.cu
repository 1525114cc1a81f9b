// Weakly-compressible SPH on the cell list: continuity, Tait pressure, Monaghan artificial
// viscosity and the symplectic Euler integrator.
//
// The reference states a pairwise equation as a gather into particle i over partners j
// (prestige/src/lib.rs:7-12 `force[i] += mass[j]`, executed by the loop of
// prestige/src/codegen/simple_cpu.rs:7-19).  These passes are that gather for the SPH rates,
// with j restricted to the particles of the neighbour cells and r_ij < 2h:
//   C_i = drho_i = sum_j m_j (v_ij . x_ij) F_ij
//   M_i = a_i    = -sum_j m_j (P_i + P_j + Pi_ij) F_ij x_ij           (+ g in the integrator)
//   F = (dW/dr)/r of the cubic spline (support 2h), P = p/rho^2, p = B((rho/rho0)^gamma - 1)
//   Pi_ij  = -2 alpha c0 h (v_ij.x_ij) / ((r^2 + eps h^2)(rho_i + rho_j))  if v_ij.x_ij < 0
//
// One time step is two passes over the same neighbour structure:
//   continuity pass  rho' = rho + dt C(x, v)   (writes rho' and P(rho') into the sorted pack)
//   momentum pass    v' = v + dt (M(x, v, rho') + g),  x' = x + dt v'   (fluid particles)
// Advancing the density first makes the acoustic pair (rho, v) symplectic; evaluating both
// rates from one snapshot would advance it by forward Euler, which amplifies every acoustic
// mode.  A third variant (pg_compute_rates) evaluates C and M of one state in one pass.
//
// Kernel structure (pg_sph_pass.cuh): the list kernel tests every candidate of the 9 (2D: 3)
// neighbour rows in FP32 against bounds on r^2, with the exact test inside their band, and
// writes each target's neighbours in walk order; the two passes evaluate the listed pairs, one
// thread per target (slot order; more in small double-word and f32 systems).  The IEEE f64 step
// evaluates each pair once instead (pg_sph_sym.cu).
// Pairs are evaluated in the oracle's order (rows z, y ascending; slots ascending), so the
// IEEE modes reproduce the oracle bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>

#include "pg_arith.cuh"
#include "pg_internal.cuh"
#include "pg_kernels.cuh"
#include "pg_sph_pass.cuh"

namespace pg {

namespace {

using namespace sphpass;

template <class R> struct V2;
template <> struct V2<double> { typedef double2 T; };
template <> struct V2<float> { typedef float2 T; };

template <class R> __device__ __forceinline__ typename V2<R>::T make2(R a, R b);
template <> __device__ __forceinline__ double2 make2<double>(double a, double b) { return make_double2(a, b); }
template <> __device__ __forceinline__ float2 make2<float>(float a, float b) { return make_float2(a, b); }

// ---------------------------------------------------------------------------------------
// Sorted gather: the final order of the neighbour search (ordered_slot), then slot k <- particle
// sorted_id[k]; precomputes P = p / rho^2.
//   f64 IEEE:  s0 {x, y, z, m}   s1 {vx, vy, vz, 0}   s2 {rho, P}   (pf: FP32 x, y, z)
//   f32:       s0 {x, y, z, m}, {vx, vy, vz, 0}   s2 {rho, P}   (pf as well)
// The f32 record is one 32-byte load per pair instead of two of 16 bytes: at 700 000 particles the
// continuity pass 0.179 -> 0.166 ms, the momentum pass 0.251 -> 0.239 ms.
// ---------------------------------------------------------------------------------------
template <class Ops, int DIM>
__global__ void sph_gather_real(SphArgs a) {
  typedef typename Ops::R R;
  typedef typename V4<R>::T R4;
  chain_begin();
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  uint32_t id;
  const uint32_t k = ordered_slot(a.order, s, id);
  const SphK& K = a.sys[sys_of_slot(a, id)];
  const R* pos = (const R*)a.pos;
  const R* vel = (const R*)a.vel;
  const R rho = ((const R*)a.rho)[id];
  const R m = ((const R*)a.mass)[id];
  R x[3] = {0, 0, 0}, v[3] = {0, 0, 0};
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    x[c] = pos[(size_t)id * DIM + c];
    v[c] = vel[(size_t)id * DIM + c];
  }
  R4 A, B;
  A.x = x[0]; A.y = x[1]; A.z = x[2]; A.w = m;
  B.x = v[0]; B.y = v[1]; B.z = v[2]; B.w = R(0);
  if (sizeof(R) == 4) {  // one 32-byte record
    ((R4*)a.s[0])[2 * (size_t)k] = A;
    ((R4*)a.s[0])[2 * (size_t)k + 1] = B;
  } else {
    ((R4*)a.s[0])[k] = A;
    ((R4*)a.s[1])[k] = B;
  }
  ((typename V2<R>::T*)a.s[2])[k] = make2<R>(rho, tait_pterm<Ops>(consts<R>(K), K.gamma, rho));
  pf_store<DIM>(a.pf, k, (float)x[0], (float)x[1], (float)x[2]);
}

// Packs of the f64 fast (double-word) mode:
//   pf x.hi, y.hi, z.hi (the list kernel's FP32 positions)
//   s0 DfHalf {x,y,z,m}.hi, {x,y,z,m}.lo (momentum pass)
//   s1 DfRecord the same and {vx,vy,vz,0}.hi, {vx,vy,vz,0}.lo (continuity pass, rates)
//   s4 {rho.hi, rho.lo, P.hi, P.lo}   s5 double {x,y,z} for the exact neighbour test near 2h.
// Positions in pf, s0 and s1 are shifted (see sph_gather_df).

// p / rho^2 of the Tait law in double-word arithmetic on the FP32 pipe (relative error about
// 1e-12: (rho/rho0)^gamma - 1 loses the digits its cancellation takes).
__device__ __forceinline__ df tait_pterm_df(const SphDF& w, int gamma, df rho) {
  const df rr = df_mul(rho, df_make(w.inv_rho0[0], w.inv_rho0[1]));
  df pw = rr;
  for (int e = 1; e < gamma; ++e) pw = df_mul(pw, rr);
  const df p = df_mul(df_make(w.B[0], w.B[1]), df_add_f(pw, -1.0f));
  return df_div(p, df_mul(rho, rho));
}

// The {rho, P/rho^2} pack of the double-word mode, from the f64 density, without FP64 work
// beyond the density itself.
__device__ __forceinline__ float4 df_pack_rho(const SphDF& w, int gamma, double rho) {
  float4 r;
  df_split_fast(rho, &r.x, &r.y);
  const df pt = tait_pterm_df(w, gamma, df_make(r.x, r.y));
  r.z = pt.hi;
  r.w = pt.lo;
  return r;
}

// The packed {rho', P'} of every slot from the canonical density, exactly as the continuity pass
// packs them (pg_step_stage: the caller may replace densities between the two passes).
template <class Ops>
__global__ void sph_repack_rho_real(SphArgs a) {
  typedef typename Ops::R R;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.n) return;
  const uint32_t id = a.sorted_id[k];
  const SphK& K = a.sys[sys_of_slot(a, id)];
  const R rn = ((const R*)a.rho)[id];
  ((typename V2<R>::T*)a.s[2])[k] = make2<R>(rn, tait_pterm<Ops>(consts<R>(K), K.gamma, rn));
}

__global__ void sph_repack_rho_df(SphArgs a) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.n) return;
  const uint32_t id = a.sorted_id[k];
  const SphK& K = a.sys[sys_of_slot(a, id)];
  ((float4*)a.s[4])[k] = df_pack_rho(K.w, K.gamma, ((const double*)a.rho)[id]);
}

// The pair passes' per-slot records in the double-word mode.  The continuity pass reads positions, mass
// and velocities (hi, lo) from one 64-byte record, half a line; the momentum pass, which needs no
// velocities, reads its own 32-byte copy of the first half: one sector, one load, and the
// records of consecutive slots, which the lanes of a warp mostly read, side by side (4M
// particles, momentum pass 2.14 ms from the 64-byte records, 1.97 from these; the gather pays 0.014
// for the copy; the continuity pass gained nothing from two 32-byte arrays).
struct __align__(32) DfHalf {
  float4 hi, lo;
};
struct __align__(64) DfRecord {
  DfHalf x, v;  // {x, y, z, m}, {vx, vy, vz, 0}
};

// Packs of the double-word mode.  Positions in the records and in the FP32 array are shifted by
// pos_pad - min (per system and dimension, pos_pad = 8h of the system), so every packed coordinate
// is at least 8h: the hi parts of two particles closer than 2h are then within a factor 2 of each
// other and the pair passes take differences with df_sub_close.  The shift is common to all
// particles of a system (pairs never cross systems), so differences are unchanged up to one f64
// rounding of each shifted coordinate, and a system's packs, hence its results, do not depend on
// the other systems of a batch; the f64 array for the exact test keeps the unshifted positions.
template <int DIM>
__global__ void sph_gather_df(SphArgs a) {
  chain_begin();
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  uint32_t id;
  const uint32_t k = ordered_slot(a.order, s, id);
  const uint32_t sys = sys_of_slot(a, id);
  const SphK& K = a.sys[sys];
  const double* pos = (const double*)a.pos;
  const double* vel = (const double*)a.vel;
  const double rho = ((const double*)a.rho)[id];
  const double m = ((const double*)a.mass)[id];
  double x[3] = {0, 0, 0}, v[3] = {0, 0, 0};
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    x[c] = pos[(size_t)id * DIM + c];
    v[c] = vel[(size_t)id * DIM + c];
  }
  double xs[3] = {K.pos_pad, K.pos_pad, K.pos_pad};
#pragma unroll
  for (int c = 0; c < DIM; ++c) xs[c] = __dadd_rn(__dsub_rn(x[c], ordered_value(a.posmin[3 * sys + c])), K.pos_pad);
  float4 ah, al, bh, bl;
  df_split_fast(xs[0], &ah.x, &al.x);
  df_split_fast(xs[1], &ah.y, &al.y);
  df_split_fast(xs[2], &ah.z, &al.z);
  df_split_fast(m, &ah.w, &al.w);
  df_split_fast(v[0], &bh.x, &bl.x);
  df_split_fast(v[1], &bh.y, &bl.y);
  df_split_fast(v[2], &bh.z, &bl.z);
  bh.w = bl.w = 0.f;
  pf_store<DIM>(a.pf, k, ah.x, ah.y, ah.z);
  DfHalf xm, vv;
  xm.hi = ah;
  xm.lo = al;
  vv.hi = bh;
  vv.lo = bl;
  DfRecord rec;
  rec.x = xm;
  rec.v = vv;
  ((DfHalf*)a.s[0])[k] = xm;
  ((DfRecord*)a.s[1])[k] = rec;
  ((float4*)a.s[4])[k] = df_pack_rho(K.w, K.gamma, rho);
  ((double4_32a*)a.s[5])[k] = make_double4_32a(x[0], x[1], x[2], 0.0);
}

// ---------------------------------------------------------------------------------------
// Pair-term policies.  STAGE: SPH_RATES (C and M of one state, written to acc/drho),
// SPH_CONT (C, then rho' = rho + dt C into the canonical state and the sorted pack),
// SPH_MOM (M with the packed rho', then the velocity and position update).
// ---------------------------------------------------------------------------------------
template <class Ops, int DIM, bool EXACT_TEST, int STAGE>
struct RealPairs {
  typedef typename Ops::R R;
  typedef typename V4<R>::T R4;
  typedef typename V2<R>::T R2;
  static constexpr bool kCont = STAGE != SPH_MOM;
  static constexpr bool kMom = STAGE != SPH_CONT;
  static constexpr bool kOneRecord = sizeof(R) == 4;  // x and v in one 32-byte record
  const R4* A;
  const R4* B;
  const R2* Q;
  SphC<R> c;
  R xi[3], vi[3], rhoi, Pi;
  R acc[3], dr;

  __device__ __forceinline__ void begin(const SphArgs& a, const SphK& K, uint32_t k) {
    A = (const R4*)a.s[0];
    B = (const R4*)a.s[1];
    Q = (const R2*)a.s[2];
    c = consts<R>(K);
    const R4 Ai = kOneRecord ? A[2 * (size_t)k] : A[k], Bi = kOneRecord ? A[2 * (size_t)k + 1] : B[k];
    xi[0] = Ai.x; xi[1] = Ai.y; xi[2] = Ai.z;
    vi[0] = Bi.x; vi[1] = Bi.y; vi[2] = Bi.z;
    rhoi = Pi = R(0);
    if (kMom) {
      const R2 q = Q[k];
      rhoi = q.x;
      Pi = q.y;
    }
    acc[0] = acc[1] = acc[2] = R(0);
    dr = R(0);
  }

  // The neighbour's pack records, loaded ahead of its pair terms.
  struct Pre {
    R4 a, b;
    R2 q;
  };
  static constexpr bool kPrefetch = true;

  __device__ __forceinline__ Pre fetch(uint32_t t, uint32_t) const {
    Pre p;
    if constexpr (kOneRecord) {
      load_32b(A + 2 * (size_t)t, p.a, p.b);
    } else {
      p.a = A[t];
      p.b = B[t];
    }
    if (kMom) p.q = Q[t];
    return p;
  }

  // A candidate of the continued walk of an overflowed list (a superset: EXACT_TEST repeats the
  // oracle's test).
  __device__ __forceinline__ void pair(uint32_t t) { terms<EXACT_TEST>(t, fetch(t, 0)); }

  // A list entry: the lists hold exactly the oracle's neighbours in every mode (f64 lists are
  // classified with the f64 test, f32 lists with the IEEE FP32 test), so no test is repeated.
  __device__ __forceinline__ void pair_with(uint32_t t, uint32_t, const Pre& p) { terms<false>(t, p); }

  // What one pair adds: dr += m w F; acc -= coef d.
  struct Term {
    R m, wF, coef, d[3];
  };

  __device__ __forceinline__ void add_term(const Term& x) {
    if (kCont) dr = Ops::add(dr, Ops::mul(x.m, x.wF));
    if (kMom) {
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) acc[cc] = Ops::sub(acc[cc], Ops::mul(x.coef, x.d[cc]));
    }
  }

  __device__ __forceinline__ void list_terms(uint32_t, uint32_t, const Pre& p, Term& x) const { evaluate<false>(p, x); }

  template <int LANES>
  static __device__ __forceinline__ Term shuffle(const Term& x, int l) {
    Term y;
    y.m = y.wF = y.coef = y.d[2] = R(0);
    if (kCont) {
      y.m = __shfl_sync(0xffffffffu, x.m, l, LANES);
      y.wF = __shfl_sync(0xffffffffu, x.wF, l, LANES);
    }
    if (kMom) {
      y.coef = __shfl_sync(0xffffffffu, x.coef, l, LANES);
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) y.d[cc] = __shfl_sync(0xffffffffu, x.d[cc], l, LANES);
    }
    return y;
  }

  template <bool TEST>
  __device__ __forceinline__ void terms(uint32_t, const Pre& p) {
    Term x;
    if (evaluate<TEST>(p, x)) add_term(x);
  }

  // false: not a neighbour (TEST).
  template <bool TEST>
  __device__ __forceinline__ bool evaluate(const Pre& p, Term& x) const {
    const R4 Aj = p.a;
    const R d0 = Ops::sub(xi[0], Aj.x), d1 = Ops::sub(xi[1], Aj.y);
    const R d2 = DIM == 3 ? Ops::sub(xi[2], Aj.z) : R(0);
    R r2 = Ops::add(Ops::mul(d0, d0), Ops::mul(d1, d1));
    if (DIM == 3) r2 = Ops::add(r2, Ops::mul(d2, d2));
    if (TEST) {
      if (!(r2 < c.four_h2)) return false;
      if (!(r2 > R(0))) return false;
    }
    const R4 Bj = p.b;
    const R r = Ops::sqrt(r2);
    const R q = Ops::mul(r, c.inv_h);
    // both pieces of the spline in the oracle's operation order, then a select (no divergence;
    // the selected value is bit for bit the oracle's)
    const R tq = Ops::sub(R(2), q);
    const R Fnear = Ops::mul(c.fa, Ops::sub(Ops::mul(R(2.25), q), R(3)));
    const R Ffar = Ops::div(Ops::mul(c.fb, Ops::mul(tq, tq)), r);
    const R F = q < R(1) ? Fnear : Ffar;
    const R dv0 = Ops::sub(vi[0], Bj.x), dv1 = Ops::sub(vi[1], Bj.y);
    const R dv2 = DIM == 3 ? Ops::sub(vi[2], Bj.z) : R(0);
    R w = Ops::add(Ops::mul(dv0, d0), Ops::mul(dv1, d1));
    if (DIM == 3) w = Ops::add(w, Ops::mul(dv2, d2));
    const R mj = Aj.w;
    if (kCont) {
      x.m = mj;
      x.wF = Ops::mul(w, F);
    }
    if (kMom) {
      const R2 qj = p.q;
      const R av = Ops::div(Ops::mul(c.avk, w), Ops::mul(Ops::add(r2, c.eps_h2), Ops::add(rhoi, qj.x)));
      const R pij = w < R(0) ? av : R(0);
      x.coef = Ops::mul(mj, Ops::mul(Ops::add(Ops::add(Pi, qj.y), pij), F));
      x.d[0] = d0;
      x.d[1] = d1;
      x.d[2] = d2;
    }
    return true;
  }

  // Sum the partial sums of the LANES lanes of a slot (butterfly; every lane ends with the sum).
  template <int LANES>
  __device__ __forceinline__ void reduce_lanes() {
#pragma unroll
    for (int off = 1; off < LANES; off <<= 1) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) acc[cc] = Ops::add(acc[cc], __shfl_xor_sync(0xffffffffu, acc[cc], off));
      dr = Ops::add(dr, __shfl_xor_sync(0xffffffffu, dr, off));
    }
  }

  __device__ __forceinline__ void finish(const SphArgs& a, const SphK& K, uint32_t id, uint32_t k) {
    if (STAGE == SPH_RATES) {
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) ((R*)a.acc)[(size_t)id * DIM + cc] = acc[cc];
      ((R*)a.drho)[id] = dr;
    } else if (STAGE == SPH_CONT) {
      R* rho = (R*)a.rho;
      const R rn = Ops::add(rho[id], Ops::mul(c.dt, dr));
      rho[id] = rn;
      ((R2*)a.s[2])[k] = make2<R>(rn, tait_pterm<Ops>(c, K.gamma, rn));
    } else if (id < K.fluid_end) {
      R* pos = (R*)a.pos;
      R* vel = (R*)a.vel;
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        const size_t o = (size_t)id * DIM + cc;
        const R v = Ops::add(vel[o], Ops::mul(c.dt, Ops::add(acc[cc], c.g[cc])));
        vel[o] = v;
        pos[o] = Ops::add(pos[o], Ops::mul(c.dt, v));
      }
    }
  }
};

template <int DIM, int STAGE>
struct DfPairs {
  static constexpr bool kCont = STAGE != SPH_MOM;
  static constexpr bool kMom = STAGE != SPH_CONT;
  const DfHalf* Xm;     // momentum pass of a step
  const DfRecord* Rec;
  const float4* RP;
  const double4_32a* Xd;
  SphDF w;
  double four_h2;
  uint32_t kself;
  float4* fc;  // per list entry {G.hi, G.lo, u.hi, u.lo} with G = m_j F and u = w / (r^2 + eps h^2):
               // written by the continuity pass, read by the momentum pass
  df xi[3], vi[3], rhoi, Pi;
  dfacc acc[3], dr;
  static constexpr bool kCacheF = STAGE == SPH_CONT || STAGE == SPH_MOM;

  __device__ __forceinline__ void begin(const SphArgs& a, const SphK& K, uint32_t k) {
    Xm = (const DfHalf*)a.s[0];
    Rec = (const DfRecord*)a.s[1];
    RP = (const float4*)a.s[4];
    Xd = (const double4_32a*)a.s[5];
    w = K.w;
    four_h2 = K.d.four_h2;
    const float4 ah = STAGE == SPH_MOM ? Xm[k].hi : Rec[k].x.hi, al = STAGE == SPH_MOM ? Xm[k].lo : Rec[k].x.lo;
    xi[0] = df_make(ah.x, al.x); xi[1] = df_make(ah.y, al.y); xi[2] = df_make(ah.z, al.z);
    if (STAGE != SPH_MOM) load_velocity(k);
    rhoi = Pi = df_make(0.f, 0.f);
    if (kMom) {
      const float4 rp = RP[k];
      rhoi = df_make(rp.x, rp.y);
      Pi = df_make(rp.z, rp.w);
    }
    kself = k;
    fc = kCacheF ? (float4*)a.fcache + list_base(k, a.cap) : nullptr;
    acc[0] = acc[1] = acc[2] = dfacc_zero();
    dr = dfacc_zero();
  }

  __device__ __forceinline__ void load_velocity(uint32_t k) {
    const float4 bh = Rec[k].v.hi, bl = Rec[k].v.lo;
    vi[0] = df_make(bh.x, bl.x); vi[1] = df_make(bh.y, bl.y); vi[2] = df_make(bh.z, bl.z);
  }

  // Geometry of pair (k, t): x_ij, r^2, F = (dW/dr)/r and w = v_ij . x_ij.  CHECK: false when t is
  // not a neighbour (outside the support, or t == k), the oracle's f64 test deciding when the
  // double-word r^2 is within a relative band of 1e-9 of (2h)^2.  Without CHECK, t comes from an
  // exact neighbour list (sph_list_kernel with f64 classification).
  // The sorted-pack records of one neighbour, loaded ahead of its pair terms.
  struct Pre {
    float4 ah, al, bh, bl, rp, fw;
  };
  static constexpr bool kPrefetch = true;
  static constexpr bool kTwo = STAGE == SPH_MOM;  // two list entries at a time (pair_two)

  __device__ __forceinline__ Pre fetch(uint32_t t, uint32_t q) const { return fetch_entry(t, q, STAGE == SPH_MOM); }

  // the momentum pass's cache entries are a DRAM stream like the lists (sph_list_pass_kernel)
  static constexpr bool kL2Entry = STAGE == SPH_MOM;
  __device__ __forceinline__ void prefetch_entry(uint32_t q) const {
    prefetch_l2(fc + (size_t)q * kListTile);
  }

  // cached: list entry q of a momentum pass that reads G = m_j F and u from the continuity pass
  __device__ __forceinline__ Pre fetch_entry(uint32_t t, uint32_t q, bool cached) const {
    Pre p;
    // the momentum pass takes w from the cache and needs no velocities of the neighbour
    load_32b(cached ? &Xm[t].hi : &Rec[t].x.hi, p.ah, p.al);
    p.bh = p.bl = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!cached) load_32b(&Rec[t].v.hi, p.bh, p.bl);
    p.rp = kMom ? RP[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    p.fw = cached ? fc[q * kListTile] : make_float4(0.f, 0.f, 0.f, 0.f);
    return p;
  }

  template <bool CHECK>
  __device__ __forceinline__ bool geometry(uint32_t t, const Pre& p, df* d, df& r2, df& F, df& wv, df& mj) const {
    const float4 ah = p.ah, al = p.al;
    d[0] = df_sub_close(xi[0], df_make(ah.x, al.x));
    d[1] = df_sub_close(xi[1], df_make(ah.y, al.y));
    d[2] = DIM == 3 ? df_sub_close(xi[2], df_make(ah.z, al.z)) : df_make(0.f, 0.f);
    r2 = df_sumsq3(d[0], d[1], d[2]);
    if (CHECK) {
      const df gap = df_sub(r2, df_make(w.four_h2[0], w.four_h2[1]));
      if (fabsf(gap.hi) <= w.band) {
        if (!exact_neighbor_call<DIM>(Xd, kself, t, four_h2)) return false;
      } else if (!(gap.hi < 0.f)) {
        return false;
      }
    }
    if (!(r2.hi > 0.f)) return false;
    const df inv_r = df_rsqrt(r2);
    // F = c0 + c1 r + c2 / r = c0 + (c1 r^2 + c2) / r on either piece of the spline, without a
    // branch and without forming r (F is continuous at r = h, so the piece chosen by the FP32
    // r^2 there does not matter beyond rounding)
    const bool near = r2.hi < w.h2;
    const df c0 = near ? df_make(w.near0[0], w.near0[1]) : df_make(w.far0[0], w.far0[1]);
    const df c1 = near ? df_make(w.near1[0], w.near1[1]) : df_make(w.far1[0], w.far1[1]);
    const df c2 = near ? df_make(0.f, 0.f) : df_make(w.far2[0], w.far2[1]);
    F = df_add_raw(c0, df_mul(df_add_raw(df_mul(c1, r2), c2), inv_r));  // consumed by products
    const float4 bh = p.bh, bl = p.bl;
    // velocity differences, consumed by the dot product only
    const df dv0 = df_sub_raw(vi[0], df_make(bh.x, bl.x));
    const df dv1 = df_sub_raw(vi[1], df_make(bh.y, bl.y));
    const df dv2 = DIM == 3 ? df_sub_raw(vi[2], df_make(bh.z, bl.z)) : df_make(0.f, 0.f);
    wv = df_dot3(dv0, dv1, dv2, d[0], d[1], d[2]);
    mj = df_make(ah.w, al.w);
    return true;
  }

  // u = w / (r^2 + eps h^2), the velocity factor of the artificial viscosity, with the sign of w
  __device__ __forceinline__ df visc_u(df r2, df wv) const {
    return df_div(wv, df_add_raw(r2, df_make(w.eps_h2[0], w.eps_h2[1])));  // a sum of positive terms
  }

  __device__ __forceinline__ df momentum_coef(const float4& rpj, df G, df u) const {
    // artificial viscosity where the pair approaches (w < 0, so u < 0), computed for every pair
    // and then selected: nearly every warp has lanes on both sides
    const df den = df_add_raw(rhoi, df_make(rpj.x, rpj.y));  // a sum of positive terms
    const df av = df_div(df_mul(df_make(w.avk[0], w.avk[1]), u), den);
    const df pij = u.hi < 0.f ? av : df_make(0.f, 0.f);
    return df_neg(df_mul(df_add_raw(df_add_raw(Pi, df_make(rpj.z, rpj.w)), pij), G));
  }

  __device__ __forceinline__ void momentum(const float4& rpj, const df* d, df G, df u) {
    const df ncoef = momentum_coef(rpj, G, u);
    dfacc_add_prod(acc[0], ncoef, d[0]);
    dfacc_add_prod(acc[1], ncoef, d[1]);
    if (DIM == 3) dfacc_add_prod(acc[2], ncoef, d[2]);
  }

  template <bool CHECK>
  __device__ __forceinline__ void terms(uint32_t t, uint32_t q, const Pre& p) {
    constexpr bool kStore = STAGE == SPH_CONT && !CHECK;  // list entries of the continuity pass
    df d[3], r2, F, wv, mj;
    if (!geometry<CHECK>(t, p, d, r2, F, wv, mj)) {
      if (kStore && fc) fc[q * kListTile] = make_float4(0.f, 0.f, 0.f, 0.f);  // contributes nothing
      return;
    }
    const df G = df_mul(mj, F);
    if (kStore && fc) {  // (fc is set; without this branch the unrolled pairs are scheduled 10 % slower)
      const df u = visc_u(r2, wv);
      fc[q * kListTile] = make_float4(G.hi, G.lo, u.hi, u.lo);
    }
    if (kCont) dfacc_add_prod(dr, G, wv);
    if (kMom) momentum(p.rp, d, G, visc_u(r2, wv));
  }

  // entry q of an exact neighbour list
  __device__ __forceinline__ void pair_with(uint32_t t, uint32_t q, const Pre& p) { terms<false>(t, q, p); }

  // What pair_with(t, q, p) adds, without adding it (sph_ordered_pass_kernel).
  static constexpr int kTerms = STAGE == SPH_MOM ? DIM : 1;
  struct Term {
    df v[kTerms];
  };
  __device__ __forceinline__ void list_terms(uint32_t t, uint32_t q, const Pre& p, Term& x) const {
    df(&out)[kTerms] = x.v;
    if constexpr (STAGE == SPH_MOM) {
      const df ncoef = momentum_coef(p.rp, df_make(p.fw.x, p.fw.y), df_make(p.fw.z, p.fw.w));
      out[0] = dfacc_term(ncoef, df_sub_close(xi[0], df_make(p.ah.x, p.al.x)));
      out[1] = dfacc_term(ncoef, df_sub_close(xi[1], df_make(p.ah.y, p.al.y)));
      if constexpr (DIM == 3) out[2] = dfacc_term(ncoef, df_sub_close(xi[2], df_make(p.ah.z, p.al.z)));
    } else {
      df d[3], r2, F, wv, mj;
      if (!geometry<false>(t, p, d, r2, F, wv, mj)) {
        fc[q * kListTile] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
      }
      const df G = df_mul(mj, F), u = visc_u(r2, wv);
      fc[q * kListTile] = make_float4(G.hi, G.lo, u.hi, u.lo);
      out[0] = dfacc_term(G, wv);
    }
  }
  __device__ __forceinline__ void add_term(const Term& x) {
#pragma unroll
    for (int c = 0; c < kTerms; ++c) dfacc_add_term(STAGE == SPH_MOM ? acc[c] : dr, x.v[c]);
  }
  template <int LANES>
  static __device__ __forceinline__ Term shuffle(const Term& x, int l) {
    Term y;
#pragma unroll
    for (int c = 0; c < kTerms; ++c)
      y.v[c] = df_make(__shfl_sync(0xffffffffu, x.v[c].hi, l, LANES), __shfl_sync(0xffffffffu, x.v[c].lo, l, LANES));
    return y;
  }
  // any candidate (the walk that continues an overflowed list): everything computed here
  __device__ __forceinline__ void pair(uint32_t t) { terms<true>(t, 0, fetch_entry(t, 0, false)); }

  // The continued walk of an overflowed list, by a policy of its own that takes the sums over and hands
  // them back, so every term is added in walk order.  Walked in the pass's own state it slowed the
  // loop over the list (4M particles, momentum pass 1.97 -> 2.7 ms).  The momentum pass evaluates
  // the rates' terms: only they read velocities, from the full records.  The continuity pass
  // reads no {rho, P}, which other threads (and the other continuity launch of the overlapped
  // schedule) are replacing.
  static constexpr bool kResumeApart = kCacheF;
  __device__ __forceinline__ void resume(const SphArgs& a, uint32_t k) {
    DfPairs<DIM, STAGE == SPH_CONT ? SPH_CONT : SPH_RATES> P;
    P.begin(a, a.sys[sys_of_slot(a, a.sorted_id[k])], k);
    P.dr = dr;
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) P.acc[cc] = acc[cc];
    continue_walk<DIM, false>(a, k, [&](uint32_t t) { P.pair(t); });
    dr = P.dr;
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) acc[cc] = P.acc[cc];
  }

  // Two list entries of the momentum pass at once, in packed arithmetic (the operations of momentum(), half a
  // for the first entry, half b for the second; without `both` the second contributes nothing).
  // Packed instructions need half the issue slots, which together with the L1's accesses limit the
  // pass: with the 32-byte records 262k particles 0.163 -> 0.131 ms, 4M 2.23 -> 1.89, 6.1M in 2D 1.15 ->
  // 0.91.  The entries' terms are added in list order, so the sums are bit for bit those of one entry
  // after the other (summing the halves apart would change the states' rounding, which the
  // mixed-precision adjoint amplifies to 2e-9 of its gradients).  The continuity pass, whose FMA
  // pipe is 67 % busy, gained nothing (262k particles 0.165 -> 0.171 to 0.188 ms).
  __device__ __forceinline__ void pair_two(const Pre& a, const Pre& b, bool both) {
    df2 d[3];
    d[0] = df2_sub_close(df2_dup(xi[0]), df2_make(f2_make(a.ah.x, b.ah.x), f2_make(a.al.x, b.al.x)));
    d[1] = df2_sub_close(df2_dup(xi[1]), df2_make(f2_make(a.ah.y, b.ah.y), f2_make(a.al.y, b.al.y)));
    d[2] = DIM == 3 ? df2_sub_close(df2_dup(xi[2]), df2_make(f2_make(a.ah.z, b.ah.z), f2_make(a.al.z, b.al.z)))
                    : df2_make(0ull, 0ull);
    const df none = df_make(0.f, 0.f);
    const df2 G = df2_pair(df_make(a.fw.x, a.fw.y), both ? df_make(b.fw.x, b.fw.y) : none);
    const df2 u = df2_make(f2_make(a.fw.z, b.fw.z), f2_make(a.fw.w, b.fw.w));
    const df2 den = df2_add_raw(df2_dup(rhoi), df2_make(f2_make(a.rp.x, b.rp.x), f2_make(a.rp.y, b.rp.y)));
    const df2 av = df2_div(df2_mul(df2_make(f2_dup(w.avk[0]), f2_dup(w.avk[1])), u), den);
    const df2 pij = df2_pair(a.fw.z < 0.f ? df2_first(av) : none, b.fw.z < 0.f ? df2_second(av) : none);
    const df2 Pj = df2_make(f2_make(a.rp.z, b.rp.z), f2_make(a.rp.w, b.rp.w));
    const df2 ncoef = df2_neg(df2_mul(df2_add_raw(df2_add_raw(df2_dup(Pi), Pj), pij), G));
    dfacc_add_prod2(acc[0], ncoef, d[0]);
    dfacc_add_prod2(acc[1], ncoef, d[1]);
    if (DIM == 3) dfacc_add_prod2(acc[2], ncoef, d[2]);
  }

  // Combine the partial sums of the LANES lanes of a slot (butterfly; every lane ends with the sum).
  template <int LANES>
  __device__ __forceinline__ void reduce_lanes() {
#pragma unroll
    for (int off = 1; off < LANES; off <<= 1) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        dfacc o;
        o.hi = __shfl_xor_sync(0xffffffffu, acc[cc].hi, off);
        o.lo = __shfl_xor_sync(0xffffffffu, acc[cc].lo, off);
        acc[cc] = dfacc_add(acc[cc], o);
      }
      dfacc o;
      o.hi = __shfl_xor_sync(0xffffffffu, dr.hi, off);
      o.lo = __shfl_xor_sync(0xffffffffu, dr.lo, off);
      dr = dfacc_add(dr, o);
    }
  }

  __device__ __forceinline__ void finish(const SphArgs& a, const SphK& K, uint32_t id, uint32_t k) {
    const SphC<double>& c = K.d;
    if (STAGE == SPH_RATES) {
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) ((double*)a.acc)[(size_t)id * DIM + cc] = dfacc_to_double(acc[cc]);
      ((double*)a.drho)[id] = dfacc_to_double(dr);
    } else if (STAGE == SPH_CONT) {
      double* rho = (double*)a.rho;
      const double rn = __dadd_rn(rho[id], __dmul_rn(c.dt, dfacc_to_double(dr)));
      rho[id] = rn;
      ((float4*)a.s[4])[k] = df_pack_rho(K.w, K.gamma, rn);
    } else if (id < K.fluid_end) {
      double* pos = (double*)a.pos;
      double* vel = (double*)a.vel;
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        const size_t o = (size_t)id * DIM + cc;
        const double v = __dadd_rn(vel[o], __dmul_rn(c.dt, __dadd_rn(dfacc_to_double(acc[cc]), c.g[cc])));
        vel[o] = v;
        pos[o] = __dadd_rn(pos[o], __dmul_rn(c.dt, v));
      }
    }
  }
};

// ---------------------------------------------------------------------------------------
// Launch plumbing: one table of kernel instantiations per (arith, dim, stage).
// ---------------------------------------------------------------------------------------
typedef void (*PassKernel)(SphArgs);

// Kernel table for the list-based passes and the list kernel (stage < 0).
template <int DIM, int STAGE, int LANES>
PassKernel list_pass_lanes(int arith) {
  switch (arith) {
    case ARITH_F64_DF: return sph_list_pass_kernel<DfPairs<DIM, STAGE>, DIM, false, LANES>;
    case ARITH_F32_FAST: return sph_list_pass_kernel<RealPairs<OpsFF, DIM, false, STAGE>, DIM, true, LANES>;
    default: return nullptr;
  }
}

template <int DIM, int STAGE>
PassKernel list_pass_for(int arith, int lanes) {
  if (lanes == 2) return list_pass_lanes<DIM, STAGE, 2>(arith);
  if (lanes == 4) return list_pass_lanes<DIM, STAGE, 4>(arith);
  switch (arith) {
    case ARITH_F64_EXACT:  // (the step's passes: pg_sph_sym.cu)
      if constexpr (STAGE == SPH_RATES) return sph_list_pass_kernel<RealPairs<OpsD, DIM, true, STAGE>, DIM, false>;
      else return nullptr;
    case ARITH_F64_DF:
      return sph_list_pass_kernel<DfPairs<DIM, STAGE>, DIM, false>;
    case ARITH_F32_EXACT:
      return sph_list_pass_kernel<RealPairs<OpsF, DIM, false, STAGE>, DIM, true>;
    case ARITH_F32_FAST:
      return sph_list_pass_kernel<RealPairs<OpsFF, DIM, false, STAGE>, DIM, true>;
    default:
      return nullptr;
  }
}

// Threads per slot of the passes of a handle of n particles with one thread per slot set: more than one
// where one would leave schedulers idle (sph_ordered_pass_kernel).  Step in us, with 1 / 2 / 4 threads
// per slot, double-word: 2D dam break of 6,518 particles 36.7 / 31.1 / 29.2, of 13,518 39.5 / 35.1 / 33.4,
// of 23,018 41.7 / 37.5 / 38.2, of 37,718 44.0 / 43.1 / 49.7; 3D lattice (half-size cells) of 5,000 particles
// 89 / 72 / 61, of 10,000 90 / 73 / 69, of 20,000 91 / 84 / 86, of 30,000 101 / 99 / 109, of 45,000
// 122 / 133 / 136.  (8 threads: 29.6 and 61.6 at the small ends, worse from there on.)  The f32 pairs
// are shorter, so the line lies higher: 3D lattice of 5,000 80 / 63 / 55, of 20,000 86 / 69 / 65, of 27,000
// 89 / 74 / 72, of 33,000 89 / 75 / 77, of 45,000 95 / 85 / 95, of 60,000 101 / 96 / 105, of 80,000
// 113 / 125 / 126 (IEEE f32 within 3 % of these).
int ordered_lanes(int arith, uint32_t n) {
  if (arith == ARITH_F64_DF) return n <= 16384 ? 4 : n <= 32768 ? 2 : 1;
  return n <= 28672 ? 4 : n <= 57344 ? 2 : 1;
}

template <int DIM, int STAGE, int LANES>
PassKernel ordered_kernel_for(int arith) {
  switch (arith) {
    case ARITH_F64_DF: return sph_ordered_pass_kernel<DfPairs<DIM, STAGE>, DIM, false, LANES>;
    case ARITH_F32_EXACT: return sph_ordered_pass_kernel<RealPairs<OpsF, DIM, false, STAGE>, DIM, true, LANES>;
    default: return sph_ordered_pass_kernel<RealPairs<OpsFF, DIM, false, STAGE>, DIM, true, LANES>;
  }
}

template <int LANES>
PassKernel ordered_kernel(int arith, int dim, int stage) {
  const bool cont = stage == SPH_CONT;
  if (dim == 2)
    return cont ? ordered_kernel_for<2, SPH_CONT, LANES>(arith) : ordered_kernel_for<2, SPH_MOM, LANES>(arith);
  return cont ? ordered_kernel_for<3, SPH_CONT, LANES>(arith) : ordered_kernel_for<3, SPH_MOM, LANES>(arith);
}

// The list kernel with the batch that suits the rows' length (see sph_list_kernel).
template <int DIM, bool EXACT_PF, int XD>
PassKernel walk_kernel(int reach) {
  if constexpr (DIM == 3) {
    if (reach == 1) return sph_list_kernel<DIM, EXACT_PF, XD, 16>;
  }
  return sph_list_kernel<DIM, EXACT_PF, XD, 8>;
}

template <int DIM>
PassKernel list_kernel_dim(int arith, int stage, int lanes, int reach) {
  switch (stage) {
    case SPH_RATES: return list_pass_for<DIM, SPH_RATES>(arith, 1);
    case SPH_CONT: return list_pass_for<DIM, SPH_CONT>(arith, lanes);
    case SPH_MOM: return list_pass_for<DIM, SPH_MOM>(arith, lanes);
    default: break;
  }
  switch (arith) {  // the list kernel
    case ARITH_F64_EXACT:  // exact lists (FP32 prefilter, the f64 test in the band): the passes skip the test
      return walk_kernel<DIM, false, 0>(reach);
    case ARITH_F64_DF:  // exact lists: the double-word passes skip the neighbour test
      return walk_kernel<DIM, false, 5>(reach);
    case ARITH_F32_EXACT:
    case ARITH_F32_FAST:
      return walk_kernel<DIM, true, -1>(reach);
    default:
      return nullptr;
  }
}

PassKernel list_kernel(int arith, int dim, int stage, int lanes, int reach) {
  lanes = sph_pass_lanes(arith, stage, lanes);
  return dim == 2 ? list_kernel_dim<2>(arith, stage, lanes, reach)
                  : list_kernel_dim<3>(arith, stage, lanes, reach);
}

// lanes: threads per slot of the kernel (1 for the list kernel); a block covers block / lanes slots.
int launch_table(cudaStream_t st, const SphArgs& a, PassKernel kern, int grid, int block, int lanes) {
  if (!kern) {
    set_error("unknown arithmetic mode or stage");
    return PG_EINVAL;
  }
  if (block < 32 || block > kSphMaxThreads || block % 32) {
    set_error("block size %d must be a multiple of 32 in 32..%d", block, kSphMaxThreads);
    return PG_EINVAL;
  }
  if (a.k_begin % (uint32_t)block || a.k_end > a.n || a.k_begin > a.k_end) {
    set_error("slot range [%u, %u) does not fit block size %d and n = %u", a.k_begin, a.k_end, block, a.n);
    return PG_EINVAL;
  }
  if (a.k_end == a.k_begin) return PG_OK;
  const uint32_t spb = (uint32_t)(block / lanes);
  const uint32_t ntiles = (a.k_end + spb - 1) / spb - a.k_begin / spb;
  if (grid <= 0 || (uint32_t)grid > ntiles) grid = (int)ntiles;
  PG_CUDA_TRY(launch_chained(st, a.chained != 0, kern, (unsigned)grid, (unsigned)block, a));
  PG_CUDA_TRY(cudaGetLastError());
  return PG_OK;
}

}  // namespace

void sph_sorted_layout(int arith, size_t sz[6]) {
  for (int i = 0; i < 6; ++i) sz[i] = 0;
  switch (arith) {
    case ARITH_F64_EXACT:  // double4 {x,m}, double4 {v,0}, double2 {rho,P}
      sz[0] = 32; sz[1] = 32; sz[2] = 16;
      break;
    case ARITH_F64_DF:  // DfHalf {x, m}, DfRecord {x, m}, {v}, float4 {rho, P} (hi, lo), double4 exact positions
      sz[0] = 32; sz[1] = 64; sz[4] = 16; sz[5] = 32;
      break;
    default:  // {float4 {x,m}, float4 {v,0}}, float2 {rho,P}
      sz[0] = 32; sz[2] = 8;
      break;
  }
}

int launch_sph_gather(cudaStream_t st, const SphArgs& a, int arith) {
  if (a.n == 0) return PG_OK;
  const unsigned blocks = (a.n + 255) / 256;
  const int dim = a.dim;
  switch (arith) {
    case ARITH_F64_EXACT:
      if (dim == 2) PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_real<OpsD, 2>, blocks, 256, a));
      else PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_real<OpsD, 3>, blocks, 256, a));
      break;
    case ARITH_F64_DF:  // a.posmin was filled by the step's hash kernel
      if (dim == 2) PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_df<2>, blocks, 256, a));
      else PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_df<3>, blocks, 256, a));
      break;
    case ARITH_F32_EXACT:
      if (dim == 2) PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_real<OpsF, 2>, blocks, 256, a));
      else PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_real<OpsF, 3>, blocks, 256, a));
      break;
    case ARITH_F32_FAST:
      if (dim == 2) PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_real<OpsFF, 2>, blocks, 256, a));
      else PG_CUDA_TRY(launch_chained(st, a.chained != 0, sph_gather_real<OpsFF, 3>, blocks, 256, a));
      break;
    default:
      set_error("unknown arithmetic mode %d", arith);
      return PG_EINVAL;
  }
  PG_CUDA_TRY(cudaGetLastError());
  return PG_OK;
}

int sph_pass_lanes(int arith, int stage, int lanes) {
  const bool tolerant = arith == ARITH_F64_DF || arith == ARITH_F32_FAST;
  return tolerant && (stage == SPH_CONT || stage == SPH_MOM) && (lanes == 2 || lanes == 4) ? lanes : 1;
}

int launch_sph_repack_rho(cudaStream_t st, const SphArgs& a, int arith) {
  if (a.n == 0) return PG_OK;
  const unsigned blocks = (a.n + 255) / 256;
  switch (arith) {
    case ARITH_F64_EXACT: sph_repack_rho_real<OpsD><<<blocks, 256, 0, st>>>(a); break;
    case ARITH_F64_DF: sph_repack_rho_df<<<blocks, 256, 0, st>>>(a); break;
    case ARITH_F32_EXACT: sph_repack_rho_real<OpsF><<<blocks, 256, 0, st>>>(a); break;
    case ARITH_F32_FAST: sph_repack_rho_real<OpsFF><<<blocks, 256, 0, st>>>(a); break;
    default:
      set_error("unknown arithmetic mode %d", arith);
      return PG_EINVAL;
  }
  PG_CUDA_TRY(cudaGetLastError());
  return PG_OK;
}

int launch_sph_list(cudaStream_t st, const SphArgs& a, int arith, int grid, int block) {
  PassKernel kern = list_kernel(arith, a.dim, -1, 1, a.reach);
  return launch_table(st, a, kern, grid, block, 1);
}

int launch_sph_list_pf(cudaStream_t st, const SphArgs& a, int grid, int block) {
  PassKernel kern = a.dim == 2 ? walk_kernel<2, false, -1>(a.reach) : walk_kernel<3, false, -1>(a.reach);
  return launch_table(st, a, kern, grid, block, 1);
}

int launch_sph_list_exact(cudaStream_t st, const SphArgs& a, int grid, int block) {
  PassKernel kern = a.dim == 2 ? walk_kernel<2, false, 0>(a.reach) : walk_kernel<3, false, 0>(a.reach);
  return launch_table(st, a, kern, grid, block, 1);
}

int launch_sph_list_pass(cudaStream_t st, const SphArgs& a, int arith, int stage, int grid, int block, int lanes) {
  lanes = sph_pass_lanes(arith, stage, lanes);
  const int ordered = arith != ARITH_F64_EXACT && lanes == 1 && stage != SPH_RATES ? ordered_lanes(arith, a.n) : 1;
  // (one block per tile)
  if (ordered == 4) return launch_table(st, a, ordered_kernel<4>(arith, a.dim, stage), 0, block, 4);
  if (ordered == 2) return launch_table(st, a, ordered_kernel<2>(arith, a.dim, stage), 0, block, 2);
  PassKernel kern = list_kernel(arith, a.dim, stage, lanes, a.reach);
  return launch_table(st, a, kern, grid, block, lanes);
}

int sph_list_regs(int arith, int dim, int reach, int stage, int lanes) {
  PassKernel kern = list_kernel(arith, dim, stage, lanes, reach);
  cudaFuncAttributes attr;
  if (!kern || cudaFuncGetAttributes(&attr, kern) != cudaSuccess) return 0;
  return attr.numRegs;
}

int sph_list_occupancy(int arith, int dim, int reach, int stage, int block, int lanes) {
  int blocks = 0;
  PassKernel kern = list_kernel(arith, dim, stage, lanes, reach);
  if (!kern) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, block, 0) != cudaSuccess) return 0;
  return blocks;
}

}  // namespace pg
