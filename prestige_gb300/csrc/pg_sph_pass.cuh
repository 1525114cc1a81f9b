// The SPH pair-pass skeleton shared by the forward passes (pg_sph.cu) and the adjoint passes
// (pg_adjoint.cu): the candidate walk over the neighbour rows with its FP32 prefilter, the
// neighbour-list kernel built on it, the list-driven pair pass (one thread per target slot) and
// the Tait pressure term.
//
// A `Pairs` policy provides
//   begin(args, system, slot)   load the target's data
//   pair(slot_j)                one candidate that passed the filter (repeats the exact test)
//   finish(args, system, id, k) write the target's results (id order; k = its slot)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pg_arith.cuh"
#include "pg_candidates.cuh"
#include "pg_internal.cuh"
#include "pg_kernels.cuh"

namespace pg {
namespace sphpass {


template <class R> struct V4;
template <> struct V4<double> { typedef double4_32a T; };
template <> struct V4<float> { typedef float4 T; };

template <class R> __device__ __forceinline__ const SphC<R>& consts(const SphK& K);
template <> __device__ __forceinline__ const SphC<double>& consts<double>(const SphK& K) { return K.d; }
template <> __device__ __forceinline__ const SphC<float>& consts<float>(const SphK& K) { return K.f; }

// p / rho^2 with p = B((rho/rho0)^gamma - 1), operation order of the oracle's tait_pterm.
template <class Ops>
__device__ __forceinline__ typename Ops::R tait_pterm(const SphC<typename Ops::R>& c, int gamma,
                                                      typename Ops::R rho) {
  typedef typename Ops::R R;
  const R rr = Ops::mul(rho, c.inv_rho0);
  R pw = rr;
  for (int e = 1; e < gamma; ++e) pw = Ops::mul(pw, rr);
  const R p = Ops::mul(c.B, Ops::sub(pw, R(1)));
  return Ops::div(p, Ops::mul(rho, rho));
}

__device__ __forceinline__ uint32_t sys_of_slot(const SphArgs& a, uint32_t id) {
  return a.sys_of_id ? a.sys_of_id[id] : 0u;
}

// ---------------------------------------------------------------------------------------
// Shared pieces of the candidate walk.
// ---------------------------------------------------------------------------------------
struct Target {
  uint32_t k, id;
  bool live;
  int cx, cy, cz, x0, x1;
};

__device__ __forceinline__ Target target_of(const SphArgs& a, uint32_t k0, const SphK** Kp, int R) {
  Target T;
  T.live = k0 < a.k_end;
  T.k = T.live ? k0 : a.n - 1;
  T.id = a.sorted_id[T.k];
  const SphK& K = a.sys[sys_of_slot(a, T.id)];
  *Kp = &K;
  const GridK& g = K.g;
  const uint32_t c = a.sorted_cell[T.k] - g.cell_base;
  T.cx = (int)(c % (uint32_t)g.nx);
  T.cy = (int)((c / (uint32_t)g.nx) % (uint32_t)g.ny);
  T.cz = (int)(c / ((uint32_t)g.nx * (uint32_t)g.ny));
  T.x0 = max(T.cx - R, 0);
  T.x1 = min(T.cx + R, g.nx - 1);
  return T;
}

// FP32 threshold on r^2.  EXACT_PF (f32 systems): the exact test.  Otherwise the conservative bound.
template <bool EXACT_PF>
__device__ __forceinline__ float prefilter_threshold(const SphK& K, const float4& pi) {
  return EXACT_PF ? K.f.four_h2 : outer_threshold(K.two_h_f, pi);
}

template <int DIM, bool EXACT_PF>
__device__ __forceinline__ bool prefilter_hit(const float4& pi, const float4& pj, float thr) {
  if (EXACT_PF) {
    const float d0 = __fsub_rn(pi.x, pj.x), d1 = __fsub_rn(pi.y, pj.y);
    float r2 = __fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1));
    if (DIM == 3) {
      const float d2 = __fsub_rn(pi.z, pj.z);
      r2 = __fadd_rn(r2, __fmul_rn(d2, d2));
    }
    return r2 < thr && r2 > 0.f;
  }
  const float d0 = pi.x - pj.x, d1 = pi.y - pj.y;
  float r2 = fmaf(d1, d1, d0 * d0);
  if (DIM == 3) {
    const float d2 = pi.z - pj.z;
    r2 = fmaf(d2, d2, r2);
  }
  return r2 < thr;
}

// The oracle's f64 neighbour test of slots k and t (positions X, double4 per slot); inline in
// the list kernel, called out of line by the pair passes (exact_neighbor_call), where the f64
// registers would otherwise count against the pair loop.
template <int DIM>
__device__ __forceinline__ bool exact_neighbor(const double4_32a* X, uint32_t k, uint32_t t, double four_h2) {
  const double4_32a xi = X[k], xj = X[t];
  const double d0 = __dsub_rn(xi.x, xj.x), d1 = __dsub_rn(xi.y, xj.y);
  double r2 = __dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1));
  if (DIM == 3) {
    const double d2 = __dsub_rn(xi.z, xj.z);
    r2 = __dadd_rn(r2, __dmul_rn(d2, d2));
  }
  return r2 < four_h2 && r2 > 0.0;
}

template <int DIM>
__device__ __noinline__ bool exact_neighbor_call(const double4_32a* X, uint32_t k, uint32_t t, double four_h2) {
  return exact_neighbor<DIM>(X, k, t, four_h2);
}

// List membership of candidate t of target k where the packed test did not decide (out of line).
// XD < 0: the FP32 test (EXACT_PF: the oracle's IEEE test, coincident positions excluded; otherwise the
// conservative prefilter, whose hits the pair passes test again).  XD >= 0: exactly the oracle's f64
// test, decided by FP32 outside its band and by the f64 positions a.s[XD] inside.
template <int DIM, bool EXACT_PF, int XD>
__device__ __noinline__ bool listed_slow(const float* PF, const double4_32a* X, uint32_t k, uint32_t t, float thr,
                                         float thr_lo, double four_h2) {
  if (t == k) return false;
  const float4 pi = pf_at<DIM>(PF, k), pj = pf_at<DIM>(PF, t);
  if (XD < 0) return prefilter_hit<DIM, EXACT_PF>(pi, pj, thr);
  const float d0 = pi.x - pj.x, d1 = pi.y - pj.y, d2 = pi.z - pj.z;
  const float r2 = DIM == 3 ? fmaf(d2, d2, fmaf(d1, d1, d0 * d0)) : fmaf(d1, d1, d0 * d0);
  if (r2 < thr_lo && r2 > 0.f) return true;
  return r2 < thr && exact_neighbor<DIM>(X, k, t, four_h2);
}

// ---------------------------------------------------------------------------------------
// Neighbour lists.  sph_list_kernel walks the candidates of every slot once per step and writes
// the listed slots (with XD < 0 the FP32 test (exact for f32 systems), with XD >= 0 exactly the
// f64 neighbours; never the slot itself) in walk order (rows z, then y ascending; slots ascending
// along a row) to nlist in warp tiles (list_base: entry q of the 32 slots of a tile is one
// 128-byte line, so a warp's reads of one entry index coalesce and its writes fill whole sectors
// while they are in L2); nlen[k] = number of listed slots (may exceed cap).  When the list fills,
// nresume[2k], [2k+1] = (row, slot) of the first listed candidate that did not fit, so the pair
// passes can continue the walk from there.
//
// Each lane walks its own rows, B candidates at a time (screen_batch: packed FP32 tests of
// consecutive slots), then stores the batch's hits in order; the lanes of a warp keep to the same
// row number, so the row bookkeeping runs once per row and warp.  What bounds it is instruction
// issue (and, through it, the latency of the loads), so the test is kept short: one sign bit per
// candidate decides, and one minimum per batch says whether every decision was certain.  The
// candidates near (2h)^2 or coincident with the target
// are decided one at a time (listed_slow).  The next batch is loaded before the hits of the
// current one are stored, the next row's slot range while the current row is walked.  Lanes whose
// targets share a cell walk the same candidates in step, so their loads coalesce (pruning each
// lane's rows to the cells its own target can reach was measured: it breaks that, and the walk got
// slower).
//
// B: long rows (3D with a reach of one cell, about 50 slots a row) take 16 candidates a batch, short
// ones (3D with a reach of two, about 11; 2D, about 17) take 8.  ms per build with 8 / 16: 3D
// 700k particles f32, reach 1 0.366 / 0.317; 262k f64, reach 2 0.113 / 0.126; 2D 6.1M 0.284 / 0.296
// (the lists of the first 70 % of the slots).
// Against the walk over {x, y, z, w} records, 16 to a batch, with two compares per candidate and
// each lane at its own row: 262k 0.153 -> 0.113 ms, f32 700k 0.412 -> 0.317, 4M (first 70 %) 1.39 -> 1.19.
// ---------------------------------------------------------------------------------------

// Offset of slot k's entry 0 in the tiled list array (entry q at + q * kListTile).
__device__ __forceinline__ size_t list_base(uint32_t k, uint32_t cap) {
  return (size_t)(k / kListTile) * cap * kListTile + (k % kListTile);
}

template <int DIM, bool EXACT_PF, int XD, int B>
__global__ void __launch_bounds__(kSphMaxThreads) sph_list_kernel(SphArgs a) {
  chain_begin();
  const int tid = threadIdx.x;
  const float* __restrict__ PF = a.pf;
  const double4_32a* __restrict__ X = (const double4_32a*)a.s[XD < 0 ? 0 : XD];
  const uint32_t* __restrict__ start = a.cell_start;
  const int R = a.reach;
  const int RZ = DIM == 3 ? R : 0;
  const int nrows = (2 * R + 1) * (2 * RZ + 1);
  const uint32_t bs = blockDim.x;
  const uint32_t tile1 = (a.k_end + bs - 1) / bs;
  constexpr unsigned kAll = (1u << B) - 1;

  for (uint32_t tile = a.k_begin / bs + blockIdx.x; tile < tile1; tile += gridDim.x) {
    const SphK* Kp;
    const Target T = target_of(a, tile * bs + tid, &Kp, R);
    const SphK& K = *Kp;
    const GridK& g = K.g;
    const float4 pi = pf_at<DIM>(PF, T.k);
    const float thr = prefilter_threshold<EXACT_PF>(K, pi);
    const float thr_lo = XD < 0 ? thr : inner_threshold(K.two_h_f, pi);
    Screen S;
    screen_target(S, pi);
    if (EXACT_PF) screen_exact(S, thr);
    else screen_band(S, thr_lo, thr);
    uint32_t* __restrict__ my = a.nlist + list_base(T.k, a.cap);  // entry q at my[q * kListTile]
    uint32_t cnt = 0;
    // The (2R + 1)^(DIM - 1) rows, z then y ascending, in step for the whole warp (the row number is
    // uniform; a row outside the grid is empty).  tn, en: the slot range of row `row + 1`.
    uint32_t tn = 0, en = 0;
    int y = T.cy - R, z = T.cz - RZ;
    uint32_t rb = row_base(g, y, z);
    auto load_range = [&]() {
      tn = en = 0;
      if (T.live && (unsigned)y < (unsigned)g.ny && (unsigned)z < (unsigned)g.nz) {
        tn = start[rb + T.x0];
        en = start[rb + T.x1 + 1];
      }
    };
    load_range();
    Batch<DIM, B> batch;
    bool loaded = false;  // batch holds the next row's first batch
    for (int row = 0; row < nrows; ++row) {
      uint32_t t = tn & ~3u;  // the batch's first slot, a multiple of 4
      const uint32_t e = tn < en ? en : 0u;
      unsigned lead = kAll >> (tn & 3u);  // valid bits of the batch's slots from the row's first on
      if (!loaded && t < e) batch.load(PF, t);
      loaded = false;
      if (row + 1 < nrows) {
        if (++y > T.cy + R) {
          y = T.cy - R;
          ++z;
          rb += ((uint32_t)g.ny - 2u * (uint32_t)R) * (uint32_t)g.nx;
        } else {
          rb += (uint32_t)g.nx;
        }
        load_range();
      } else {
        tn = en = 0;
      }
      while (t < e) {
        // the batch's candidates that belong to the row, the target itself left out
        unsigned valid = lead;
        if (e - t < (uint32_t)B) valid &= ~(kAll >> (e - t));
        if (T.k - t < (uint32_t)B) valid &= ~((kAll + 1) / 2 >> (T.k - t));
        unsigned open;
        unsigned hit = screen_batch<DIM, B, !EXACT_PF, !EXACT_PF>(batch, S, open) & valid;
        const uint32_t first = t;
        lead = kAll;
        t += B;
        // the next batch (of this row, or the next row's first), in flight while the hits are stored
        loaded = t >= e && tn < en;
        if (t < e || loaded) batch.load(PF, t < e ? t : tn & ~3u);
        open &= valid;
        for (hit &= ~open; open; open &= open - 1) {
          const int b = B - __ffs(open);
          if (listed_slow<DIM, EXACT_PF, XD>(PF, X, T.k, first + b, thr, thr_lo, K.d.four_h2)) hit |= open & -open;
        }
        if (!hit) continue;
        const uint32_t end = cnt + __popc(hit);
        if (end <= a.cap) {
          uint32_t* __restrict__ out = my + (size_t)cnt * kListTile;
#pragma unroll
          for (int b = 0; b < B; ++b)
            if (hit >> (B - 1 - b) & 1u) {
              *out = first + b;
              out += kListTile;
            }
        } else {  // the list is full, or becomes so within this batch
          for (uint32_t q = cnt; hit; ++q) {
            const int b = 31 - __clz(hit);
            hit ^= 1u << b;
            const uint32_t c = first + B - 1 - b;
            if (q < a.cap) {
              my[(size_t)q * kListTile] = c;
            } else if (q == a.cap) {
              a.nresume[2 * (size_t)T.k] = (uint32_t)row;
              a.nresume[2 * (size_t)T.k + 1] = c;
            }
          }
        }
        cnt = end;
      }
    }
    if (T.live) a.nlen[T.k] = cnt;
  }
}

// ---------------------------------------------------------------------------------------
// Mirror entries of the pair-once kernels: the position of a slot in another slot's stored list
// (lists ascend).
// ---------------------------------------------------------------------------------------
constexpr uint32_t kNoMirror = 0xFFFFFFFFu;
constexpr int kSearch = 4;  // searches in flight per thread

// First of the L entries of an ascending tiled list that is not below k.
__device__ __forceinline__ uint32_t lower_bound(const uint32_t* __restrict__ list, uint32_t L, uint32_t k) {
  uint32_t lo = 0, hi = L;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (list[(size_t)mid * kListTile] < k) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// pos[i] = position of slot k in the stored list of slot t[i], or kNoMirror.  The searches run in step, so
// each round has kSearch loads in flight in place of one.
__device__ __forceinline__ void find_in_lists(const SphArgs& a, const uint32_t (&t)[kSearch], uint32_t k,
                                              uint32_t (&pos)[kSearch]) {
  uint32_t hi[kSearch], L[kSearch];
  const uint32_t* lt[kSearch];
  bool more = false;
#pragma unroll
  for (int i = 0; i < kSearch; ++i) {
    L[i] = hi[i] = min(a.nlen[t[i]], a.cap);
    lt[i] = a.nlist + list_base(t[i], a.cap);
    pos[i] = 0;
    more = more || hi[i] > 0;
  }
  while (more) {
    more = false;
    uint32_t v[kSearch], mid[kSearch];
#pragma unroll
    for (int i = 0; i < kSearch; ++i) {
      mid[i] = (pos[i] + hi[i]) >> 1;
      v[i] = pos[i] < hi[i] ? lt[i][(size_t)mid[i] * kListTile] : 0u;
    }
#pragma unroll
    for (int i = 0; i < kSearch; ++i) {
      if (pos[i] < hi[i]) {
        if (v[i] < k) pos[i] = mid[i] + 1;
        else hi[i] = mid[i];
      }
      more = more || pos[i] < hi[i];
    }
  }
#pragma unroll
  for (int i = 0; i < kSearch; ++i)
    if (pos[i] >= L[i] || lt[i][(size_t)pos[i] * kListTile] != k) pos[i] = kNoMirror;
}

// What the pair-once kernels keep of entry j above slot k, in one word: the mirror index (13 bits, all ones
// for none; a list holds at most 4096 entries) and the partner as its distance from k (19 bits; all
// ones: read it from the list).  Partners farther apart in slot order need a row or plane of cells of
// half a million particles; the distance spares the others a read of the list at 32 scattered places
// per warp.  1M particles, IEEE: six steps with host copies 26.5 ms, with two words 27.9.
constexpr uint32_t kNoPos = 0x1fffu, kFar = 0x7ffffu;
struct Mirror {
  uint32_t pos, slot;
};
__device__ __forceinline__ uint32_t mirror_word(uint32_t pos, uint32_t slot, uint32_t k) {
  return pos << 19 | min(slot - k, kFar);  // (kNoMirror becomes kNoPos)
}
// upper: the slot's list from its first entry above the slot
__device__ __forceinline__ Mirror mirror_of(uint32_t word, uint32_t k, const uint32_t* __restrict__ upper, uint32_t j) {
  Mirror m;
  m.pos = word >> 19;
  const uint32_t d = word & kFar;
  m.slot = d != kFar ? k + d : upper[(size_t)j * kListTile];
  return m;
}

// 32 bytes from a 32-byte aligned address by one load per lane (read-only for the kernel).
__device__ __forceinline__ void load_32b(const float4* p, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// L2 prefetch hint for one address (PTX prefetch.global.L2; a hint, it returns nothing).
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// List entries (and, for policies with kL2Entry, the policy's own per-entry data through
// prefetch_entry(q)) are prefetched into L2 this many entries ahead of their use: both are
// streams from DRAM, read once, that the one-entry-ahead register prefetch cannot cover.
constexpr uint32_t kL2Ahead = 8;

template <class P, class = void>
struct L2EntryPolicy {
  static constexpr bool value = false;
};
template <class P>
struct L2EntryPolicy<P, decltype((void)P::kL2Entry)> {
  static constexpr bool value = P::kL2Entry;
};

// Policies that split a pair into fetch(t, q) (the loads for neighbour t, entry q of the list) and
// pair_with(t, q, fetched).
template <class P, class = void>
struct PrefetchPolicy {
  static constexpr bool value = false;
};
template <class P>
struct PrefetchPolicy<P, decltype((void)P::kPrefetch)> {
  static constexpr bool value = P::kPrefetch;
};

// The rest of the candidate walk of slot k after its list reached capacity, in walk order: fn(t) for every
// candidate that passes the FP32 test.
template <int DIM, bool EXACT_PF, class Fn>
__device__ __forceinline__ void continue_walk(const SphArgs& a, uint32_t k, Fn&& fn) {
  const SphK* Kp;
  const Target T = target_of(a, k, &Kp, a.reach);
  const SphK& K = *Kp;
  const GridK& g = K.g;
  const int R = a.reach, RZ = DIM == 3 ? R : 0, side = 2 * R + 1, nrows = side * (2 * RZ + 1);
  const float4 pi = pf_at<DIM>(a.pf, k);
  const float thr = prefilter_threshold<EXACT_PF>(K, pi);
  const int row0 = (int)a.nresume[2 * (size_t)k];
  const uint32_t t0 = a.nresume[2 * (size_t)k + 1];
  for (int row = row0; row < nrows; ++row) {
    const int z = T.cz + row / side - RZ, y = T.cy + row % side - R;
    if (z < 0 || z >= g.nz || y < 0 || y >= g.ny) continue;
    const uint32_t rb = row_base(g, y, z);
    const uint32_t e = a.cell_start[rb + T.x1 + 1];
    for (uint32_t t = row == row0 ? t0 : a.cell_start[rb + T.x0]; t < e; ++t)
      if (prefilter_hit<DIM, EXACT_PF>(pi, pf_at<DIM>(a.pf, t), thr)) fn(t);
  }
}

// Policies that sum the continued walk apart: resume(args, slot).
template <class P, class = void>
struct ResumePolicy {
  static constexpr bool value = false;
};
template <class P>
struct ResumePolicy<P, decltype((void)P::kResumeApart)> {
  static constexpr bool value = P::kResumeApart;
};

// Policies whose passes take two entries at a time: pair_two(fetched a, fetched b, both).
template <class P, class = void>
struct TwoPolicy {
  static constexpr bool value = false;
};
template <class P>
struct TwoPolicy<P, decltype((void)P::kTwo)> {
  static constexpr bool value = P::kTwo;
};

// Pair pass over the lists of sph_list_kernel (any block size up to kSphMaxThreads, a
// multiple of 32).  LANES consecutive threads share one target slot (32 / LANES particles per
// warp): lane `sub` of a slot takes its list entries sub, sub + LANES, ..., the lanes' partial
// sums are combined by the policy's reduce_lanes<LANES>() (a fixed butterfly, so the result is
// deterministic) and lane 0 writes the slot's results.  LANES > 1 changes the summation order,
// so only the tolerance-based modes (double-word f64, contracted f32) use it.  Lanes step
// through their lists together; a list that overflowed is followed by the rest of the walk from
// its resume point (lane 0).
template <class Pairs, int DIM, bool EXACT_PF, int LANES = 1>
__global__ void __launch_bounds__(kSphMaxThreads) sph_list_pass_kernel(SphArgs a) {
  static_assert(LANES == 1 || LANES == 2 || LANES == 4, "1, 2 or 4 lanes per slot");
  chain_begin();
  const int tid = threadIdx.x;
  const uint32_t cap = a.cap;
  const uint32_t spb = blockDim.x / LANES;  // slots per block
  const uint32_t sub = LANES > 1 ? (uint32_t)tid % LANES : 0u;
  const uint32_t tile1 = (a.k_end + spb - 1) / spb;
  for (uint32_t tile = a.k_begin / spb + blockIdx.x; tile < tile1; tile += gridDim.x) {
    const uint32_t k0 = tile * spb + (uint32_t)tid / LANES;
    const bool live = k0 < a.k_end;
    const uint32_t k = live ? k0 : a.n - 1;
    const uint32_t id = a.sorted_id[k];
    const SphK& K = a.sys[sys_of_slot(a, id)];
    Pairs P;
    P.begin(a, K, k);
    const uint32_t cnt = live ? a.nlen[k] : 0u;
    const uint32_t L = min(cnt, cap);
    const uint32_t* __restrict__ my = a.nlist + list_base(k, cap);  // entry q at my[q * kListTile]
    if constexpr (TwoPolicy<Pairs>::value) {
      // software pipeline over pairs of entries: list entries two pairs ahead, records one
      constexpr uint32_t S = LANES;
      auto at = [&](uint32_t q) { return my[(size_t)min(q, L - 1) * kListTile]; };
      if (sub < L) {
        uint32_t tna = at(sub + 2 * S), tnb = at(sub + 3 * S);
        typename Pairs::Pre ca = P.fetch(at(sub), sub), cb = P.fetch(at(sub + S), min(sub + S, L - 1));
        for (uint32_t q = sub; q < L; q += 2 * S) {
          if (q + kL2Ahead * S < L) {
            prefetch_l2(my + (size_t)(q + kL2Ahead * S) * kListTile);
            prefetch_l2(my + (size_t)min(q + (kL2Ahead + 1) * S, L - 1) * kListTile);
            if constexpr (L2EntryPolicy<Pairs>::value) {
              P.prefetch_entry(q + kL2Ahead * S);
              P.prefetch_entry(min(q + (kL2Ahead + 1) * S, L - 1));
            }
          }
          const uint32_t ta = at(q + 4 * S), tb = at(q + 5 * S);
          const typename Pairs::Pre na = P.fetch(tna, min(q + 2 * S, L - 1)), nb = P.fetch(tnb, min(q + 3 * S, L - 1));
          P.pair_two(ca, cb, q + S < L);
          ca = na;
          cb = nb;
          tna = ta;
          tnb = tb;
        }
      }
    } else if constexpr (PrefetchPolicy<Pairs>::value) {
      // software pipeline: list entries two ahead, the neighbour's pack records one ahead; the
      // unrolled pair bodies (branch-free) interleave
      constexpr uint32_t S = LANES;
      const uint32_t q0 = sub;
      uint32_t t = q0 < L ? my[q0 * kListTile] : k;
      uint32_t tn = q0 + S < L ? my[(q0 + S) * kListTile] : t;
      typename Pairs::Pre cur = P.fetch(t, q0 < L ? q0 : 0);
#pragma unroll 2
      for (uint32_t q = q0; q < L; q += S) {
        if (q + kL2Ahead * S < L) {
          prefetch_l2(my + (size_t)(q + kL2Ahead * S) * kListTile);
          if constexpr (L2EntryPolicy<Pairs>::value) P.prefetch_entry(q + kL2Ahead * S);
        }
        const uint32_t tnn = q + 2 * S < L ? my[(q + 2 * S) * kListTile] : tn;
        const typename Pairs::Pre nxt = P.fetch(tn, q + S < L ? q + S : q);
        P.pair_with(t, q, cur);
        cur = nxt;
        t = tn;
        tn = tnn;
      }
    } else {
      for (uint32_t q = sub; q < L; q += LANES) P.pair(my[q * kListTile]);
    }
    if (cnt > cap && sub == 0) {  // rare: continue the candidate walk where the list stopped
      if constexpr (ResumePolicy<Pairs>::value) P.resume(a, k);
      else continue_walk<DIM, EXACT_PF>(a, k, [&](uint32_t t) { P.pair(t); });
    }
    if constexpr (LANES > 1) P.template reduce_lanes<LANES>();  // whole warps: the tile loop is uniform
    if (live && sub == 0) P.finish(a, K, id, k);
  }
}

// The pass with LANES threads per slot for systems that leave the chip idle: a slot's pairs are
// evaluated LANES at a time, and every lane then adds the LANES terms in list order (shuffled from the
// lane that has them), so the sums are bit for bit those of one thread per slot.  What bounds such a
// system is the chain of one thread's pairs, each a few hundred dependent instructions; the additions are
// a tenth of them.  One block per tile.
template <class Pairs, int DIM, bool EXACT_PF, int LANES>
__global__ void __launch_bounds__(kSphMaxThreads) sph_ordered_pass_kernel(SphArgs a) {
  chain_begin();
  const uint32_t cap = a.cap, sub = threadIdx.x % LANES, spb = blockDim.x / LANES;
  const uint32_t k0 = (a.k_begin / spb + blockIdx.x) * spb + threadIdx.x / LANES;
  const bool live = k0 < a.k_end;
  const uint32_t k = live ? k0 : a.n - 1;
  const uint32_t id = a.sorted_id[k];
  const SphK& K = a.sys[sys_of_slot(a, id)];
  Pairs P;
  P.begin(a, K, k);
  const uint32_t cnt = live ? a.nlen[k] : 0u;
  const uint32_t L = min(cnt, cap), longest = __reduce_max_sync(0xffffffffu, L);
  const uint32_t* __restrict__ my = a.nlist + list_base(k, cap);
  auto at = [&](uint32_t q) { return q < L ? my[(size_t)q * kListTile] : k; };
  uint32_t t = at(sub), tn = at(sub + LANES);
  typename Pairs::Pre cur = P.fetch(t, sub < L ? sub : 0u);
  for (uint32_t q0 = 0; q0 < longest; q0 += LANES) {
    const uint32_t q = q0 + sub, tnn = at(q + 2 * LANES);
    const typename Pairs::Pre nxt = P.fetch(tn, q + LANES < L ? q + LANES : 0u);
    typename Pairs::Term term = {};  // adds nothing
    if (q < L) P.list_terms(t, q, cur, term);
#pragma unroll
    for (int l = 0; l < LANES; ++l) P.add_term(Pairs::template shuffle<LANES>(term, l));
    cur = nxt;
    t = tn;
    tn = tnn;
  }
  if (cnt > cap && sub == 0) {  // rare: continue the candidate walk where the list stopped
    if constexpr (ResumePolicy<Pairs>::value) P.resume(a, k);
    else continue_walk<DIM, EXACT_PF>(a, k, [&](uint32_t tt) { P.pair(tt); });
  }
  if (live && sub == 0) P.finish(a, K, id, k);
}

}  // namespace sphpass
}  // namespace pg
