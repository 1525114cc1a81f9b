// Internal declarations of the GB300 (sm_103a) particle library.
//
// Data layout in HBM (one handle = one particle system, or a batch of independent systems
// concatenated in id order):
//   canonical state, particle-id order   pos[n*dim], vel[n*dim], rho[n], mass[n]   (SPH)
//                                        pos, vel, omega[n*3], radius[n], mass[n]  (DEM)
//   neighbour search, every step         cell of each id -> stable counting sort by cell
//                                        -> sorted_cell[k], sorted_id[k] (slot k)
//                                        cell_start[c], n_cells + 1 entries
//   sorted packed copies, slot order     read by the pair kernels (coalesced, shared in L1)
// The pair kernels read only the sorted copies and write the canonical entries of their own
// particle, so one launch holds both the force loop and the integrator.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/prestige_gpu.h"

namespace pg {

// ---------------------------------------------------------------------------------------
// Errors: a thread-local message plus an integer status.
// ---------------------------------------------------------------------------------------
void set_error(const char* fmt, ...);
void clear_error();
const char* last_error();

#define PG_CUDA_TRY(expr)                                                                            \
  do {                                                                                               \
    cudaError_t e_ = (expr);                                                                         \
    if (e_ != cudaSuccess) {                                                                         \
      ::pg::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__);   \
      return e_ == cudaErrorMemoryAllocation ? PG_ENOMEM : PG_ECUDA;                                 \
    }                                                                                                \
  } while (0)

#define PG_TRY(expr)            \
  do {                          \
    int s_ = (expr);            \
    if (s_ != PG_OK) return s_; \
  } while (0)

// Device error word bits (set with atomicOr by kernels, read at synchronisation points).
enum : unsigned {
  ERR_CONTACT_OVERFLOW = 1u,  // DEM: a particle had more contacts than history slots
};

// ---------------------------------------------------------------------------------------
// Dependent launches inside a step and from one step to the next.  The kernels of a step form a chain on
// one stream, and below about 100k particles a good part of a step is the gap between a kernel's end
// and the next one's first instruction.  A kernel launched with launch_chained directly after another
// kernel (no copy, memset or event in between) is set up while that one runs and starts as its last
// blocks end; chain_begin(), first in every kernel that is launched so, waits until the earlier kernel
// is complete and its writes are visible.  Since every kernel waits for the one before, a kernel's inputs may come from
// any earlier kernel of the stream.  us per step with plain and chained launches: dam break, 6.5k
// particles, eager 51.8 / 38.0, as a graph 38.8 / 37.2; 100k eager 244 / 231; 262k eager 475 / 463.
// The first kernel of a step is chained to the step before it: 3D lattice of 5,000 particles, eager, 61.5 -> 59.4.
// Letting the next kernel's blocks in from the start of the current one (an early launch_dependents)
// was slower (100k 273, 262k 489): they settle unevenly over the SMs.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
cudaError_t launch_chained(cudaStream_t st, bool chained, void (*kernel)(P...), unsigned grid, unsigned block,
                           A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// ---------------------------------------------------------------------------------------
// Owned device buffer.  Allocated at set-up only, never inside a step, so a step can be
// captured into a CUDA graph.
// ---------------------------------------------------------------------------------------
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void release();
  int ensure(size_t nbytes);  // grow to at least nbytes (contents undefined after growth)
  template <class T> T* as() const { return (T*)p; }
};

// ---------------------------------------------------------------------------------------
// Cell grid.  Cell side s = mult * support * (1 + 2^-20); the inflation keeps every pair
// closer than `support` within `reach` cells after rounding.  Cell index
// c = (cz * ny + cy) * nx + cx with c_d = clamp(floor((x_d - lo_d) * inv), 0, n_d - 1),
// evaluated as one IEEE subtraction then one multiplication in the system precision.
// Clamping is monotone, so particles outside the box still find every neighbour.
// ---------------------------------------------------------------------------------------
struct Grid {
  int dim = 3;
  double lo[3] = {0, 0, 0};
  double cell = 1.0, inv = 1.0, support = 1.0;
  int n[3] = {1, 1, 1};
  int reach = 1;
  uint64_t ncells() const { return (uint64_t)n[0] * n[1] * n[2]; }
};
int make_grid(int dim, const double lo[3], const double hi[3], double support, double mult, Grid* g);

// Kernel-side copy of a grid.
struct GridK {
  double lo[3];
  double inv;
  double support;
  float lof[3];
  float invf;
  float support_f;
  int nx, ny, nz;
  int reach;
  int dim;
  uint32_t cell_base;  // added to every cell index (batched systems)
};
GridK grid_k(const Grid& g, uint32_t cell_base);

// Index of the first cell of row (y, z).  Unsigned: a grid may have almost 2^32 cells, and the walks form the
// bases of rows outside the grid too (such a value wraps and is not read).
__host__ __device__ __forceinline__ uint32_t row_base(const GridK& g, int y, int z) {
  return g.cell_base + ((uint32_t)z * (uint32_t)g.ny + (uint32_t)y) * (uint32_t)g.nx;
}

// The slot (from 0) of a thread where LANES consecutive threads share one (block: a multiple of LANES).  Not
// the thread's number in the grid divided by LANES: that number has 34 bits at 2^32 slots.
template <int LANES>
__host__ __device__ __forceinline__ uint32_t lane_slot(uint32_t block_id, uint32_t block, uint32_t thread) {
  return block_id * (block / LANES) + thread / LANES;
}

// ---------------------------------------------------------------------------------------
// Neighbour-search workspace: stable sort of the particles by cell, and the cell table (pg_sort.cu).
// ---------------------------------------------------------------------------------------
constexpr uint32_t kScanChunk = 8192;  // cells a block of the scan takes at a time
constexpr uint32_t kBigCell = 1024;    // larger cells are ranked by tiles of ids (see pg_sort.cu)
constexpr uint32_t kMaxTiles = 1024;

// What the hash gives the sort beside the cells.
enum HashMode {
  HASH_COUNT,         // counting sort: arrival ranks, an atomic per particle
  HASH_COUNT_MERGED,  // the same, one atomic for a warp's particles of a cell
  HASH_IDS,           // radix sort: ids
};

struct NbrWork {
  size_t n = 0;
  uint64_t ncells = 0;
  HashMode mode = HASH_COUNT;
  bool radix = false;  // mode == HASH_IDS
  int passes = 0;      // 8-bit digits of a cell index
  DevBuf mem;          // all arrays below
  uint32_t *sorted_cell = nullptr, *sorted_id = nullptr;  // [n] cell and id of each sorted slot
  uint32_t* cell_start = nullptr;                         // [ncells + 1], padded to whole chunks
  uint32_t *key = nullptr, *rank = nullptr;  // [n] cell and arrival rank of each id (radix: cells and ids to sort)
  // counting sort
  uint32_t chunks = 0;              // scan chunks: cover ncells + 1 entries
  uint32_t* unsorted = nullptr;     // [n] ids by cell
  uint32_t* chunk_total = nullptr;  // [chunks] particles per block of the scan
  uint32_t* tile_count = nullptr;   // cells of more than kBigCell: rows of tile_row words (see pg_sort.cu)
  uint32_t tile_fine = 0, tile_row = 0;
  int tile_shift = 0;               // log2 of the ids per tile
  uint32_t* rest = nullptr;         // the arrays that are zero between searches, rest_words in all:
  uint32_t* count = nullptr;        //   [chunks * kScanChunk] particles per cell
  uint32_t* big = nullptr;          //   {1 where a cell holds more than kBigCell, blocks done}
  size_t rest_words = 0;
  // radix sort
  uint32_t *key2 = nullptr, *id2 = nullptr;  // [n]
  uint32_t *hist = nullptr, *digit_total = nullptr;
  int tiles = 0;

  bool clean = false;  // count, big and the position minima hold their rest values
  int init(size_t n, uint64_t ncells);
  size_t bytes() const;
  int launches() const { return radix ? 2 + 3 * passes : chunks > 1 ? 4 : 3; }  // of one search
};

// What a sorted-gather kernel needs to finish the sort: ordered_slot() gives each thread the particle
// and the final slot of one entry of `unsorted`, and records both.
struct NbrOrder {
  const uint32_t* unsorted;
  const uint32_t* key;  // null: sorted already, `unsorted` being sorted_id
  const uint32_t* cell_start;
  uint32_t* sorted_cell;
  uint32_t* sorted_id;
  const uint32_t* rank;
  const uint32_t* tile_count;
  uint32_t tile_fine, tile_row;
  int tile_shift;
};
NbrOrder nbr_order(const NbrWork& w);

// Members of a cell (slots [b, e), more than 32) with smaller ids: counted four ids a load, or in cells of more
// than kBigCell the id's rank in its tile plus the counts of the tiles before (pg_sort.cu).  Out of
// line, so the gathers of ordinary cells do not hold it.
static __device__ __noinline__ uint32_t large_cell_rank(const uint32_t* unsorted, const uint32_t* rank,
                                                        const uint32_t* tile_count, uint32_t tile_fine,
                                                        uint32_t tile_row, int tile_shift, uint32_t id, uint32_t b,
                                                        uint32_t e) {
  uint32_t k = 0;
  if (e - b <= kBigCell) {
    uint32_t q = b;
    for (; q & 3u; ++q) k += unsorted[q] < id ? 1u : 0u;
    for (; q + 4 <= e; q += 4) {  // four ids a load
      const uint4 v = *(const uint4*)(unsorted + q);
      k += (v.x < id ? 1u : 0u) + (v.y < id ? 1u : 0u) + (v.z < id ? 1u : 0u) + (v.w < id ? 1u : 0u);
    }
    for (; q < e; ++q) k += unsorted[q] < id ? 1u : 0u;
    return k;
  }
  k = rank[id];
  const uint32_t* row = tile_count + (size_t)(b / kBigCell) * tile_row;
  const uint32_t tile = id >> tile_shift;
  for (uint32_t g = 0; g < tile / 32; ++g) k += row[tile_fine + g];
  for (uint32_t t = tile & ~31u; t < tile; ++t) k += row[t];
  return k;
}

// Within a cell the scatter left the ids in arrival order: an id's slot is the cell's first plus the
// number of smaller ids in the cell, so equal cells end up in id order (the stable order).
__device__ __forceinline__ uint32_t ordered_slot(const NbrOrder& o, uint32_t s, uint32_t& id) {
  id = o.unsorted[s];
  if (!o.key) return s;
  const uint32_t c = o.key[id];
  const uint32_t b = o.cell_start[c], e = o.cell_start[c + 1];
  uint32_t k = b;
  if (e - b <= 32)
    for (uint32_t q = b; q < e; ++q) k += o.unsorted[q] < id ? 1u : 0u;
  else
    k += large_cell_rank(o.unsorted, o.rank, o.tile_count, o.tile_fine, o.tile_row, o.tile_shift, id, b, e);
  o.sorted_id[k] = id;
  o.sorted_cell[k] = c;
  return k;
}

// Cell of every particle (id order) with its arrival rank in the cell, counted into w.count (radix sort:
// with its id).
// posmin (optional, f64 positions only): per system and dimension ([3 sys + d]) the minimum
// position, as ordered_code values, folded in with atomicMin (all ones before).
// chained: directly after another kernel of the stream.
int launch_hash(cudaStream_t st, bool chained, const GridK* grid_dev, const uint32_t* sys_of_id, int f64, int dim,
                const void* pos, NbrWork& w, unsigned long long* posmin = nullptr);

// Order-preserving map of doubles to unsigned 64-bit integers (and back), for atomicMin.
__device__ __forceinline__ unsigned long long ordered_code(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ordered_value(unsigned long long u) {
  return __longlong_as_double((long long)((u >> 63) ? (u & 0x7fffffffffffffffull) : ~u));
}
// Cell table and the ids grouped by cell, from launch_hash's arrays; the sorted gather that follows
// orders the ids within each cell (ordered_slot).  nmin position minima move from minacc to minout
// (both optional), minacc going back to all ones.
int launch_sort(cudaStream_t st, NbrWork& w, unsigned long long* minacc, unsigned long long* minout, uint32_t nmin);
// Exclusive scan of m u32 values into out[0..m] (out[m] = total).  tmp: scan_tmp_words(m).
size_t scan_tmp_words(size_t m);
int launch_exclusive_scan(cudaStream_t st, const uint32_t* in, uint32_t* out, size_t m, uint32_t* tmp);

}  // namespace pg
