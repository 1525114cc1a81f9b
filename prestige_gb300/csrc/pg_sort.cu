// Neighbour-search integer stages: device exclusive scan, stable counting sort of the particles by
// cell with its cell-start table, and the radix sort of the cell list without allocation.
//
// The reference executes an equation as `for i in 0..n { for j in 0..n { body } }`
// (prestige/src/codegen/simple_cpu.rs:7-8).  These stages replace the inner all-pairs loop
// by a cell list: particles are ordered by (cell, id) and cell c owns the slots
// cell_start[c] .. cell_start[c+1].  Everything here is integer work and bit-exact against
// the oracle's stable counting sort.
//
// The sort of a handle takes three or four launches and a share of the sorted gather that follows:
//   hash (pg_neighbors.cu)  cell of each id; an atomic on the cell's count gives the id its arrival
//                rank there
//   cell_reduce  totals per block of the scan (grids of more than one chunk of kScanChunk cells; adding them up by
//                atomics in the hash took 5 ns per warp of particles: one address at a time)
//   cell_scan    cell_start = exclusive scan of the counts: a block per chunk (in the largest grids for
//                several), its base the sum of the totals of the blocks before it; the counts go
//                back to zero for the next search
//   cell_scatter id -> slot cell_start[cell] + rank, so ids are grouped by cell in arrival order
//   the gather   ranks each id among the ids of its cell (ordered_slot): the stable order
// It is bound by the latency of these few launches below about 1M particles and by the scattered
// 4-byte writes and atomics above.  Search plus gather, ms, by the radix sort below and by this one:
// 6.5k particles 0.049 / 0.025, 200k spheres 0.085 / 0.045, 262k 0.082 / 0.041, 700k f32
// 0.073 / 0.050, 4M 0.409 / 0.254, 6.1M in 512 systems 0.589 / 0.401.
//
// Ranking an id among the m ids of its cell takes the gather m reads.  Cells of more than kBigCell
// particles take counts per tile of consecutive ids instead: rank = rank within the tile + the counts of
// the tiles before (rank_big_cells, large_cell_rank).  Search of 1M particles in 100 of 10,000 cells 0.35 ms; one
// block that sorts such cells one after the other takes 8.5, the radix sort about 0.1.  Dense grids take
// an LSD radix sort (sort_mode).
#include <cuda_runtime.h>

#include <mutex>
#include <utility>

#include "pg_internal.cuh"

namespace pg {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;  // keys per thread of the radix kernels: their scratch has a fixed size
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096 keys per tile
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kRadix = 256;

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096 values per block

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x multiple of 32, <= 1024).
// Returns the exclusive prefix; *total receives the block sum.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t block_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint32_t incl = warp_incl_scan(v);
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < nwarps ? warp_sums[lane] : 0u;
    uint32_t si = warp_incl_scan(s);
    if (lane < nwarps) warp_sums[lane] = si - s;
    if (lane == nwarps - 1) block_total = si;
  }
  __syncthreads();
  uint32_t r = incl - v + warp_sums[warp];
  if (total) *total = block_total;
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------------------------------
// Exclusive scan (reduce, scan block sums, rescan).  out[m] receives the total.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ in, size_t m,
                                                                   uint32_t* __restrict__ bsum) {
  const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < m) s += in[base + k];
  uint32_t total;
  block_excl_scan(s, &total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// One block scans the block sums sequentially in chunks of kScanThreads (any count).
__global__ void __launch_bounds__(kScanThreads) scan_bsum_kernel(uint32_t* __restrict__ bsum, size_t nb) {
  uint32_t carry = 0;
  for (size_t c0 = 0; c0 < nb; c0 += kScanThreads) {
    const size_t i = c0 + threadIdx.x;
    uint32_t v = i < nb ? bsum[i] : 0u;
    uint32_t total;
    uint32_t ex = block_excl_scan(v, &total);
    if (i < nb) bsum[i] = ex + carry;
    carry += total;
  }
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const uint32_t* __restrict__ in, size_t m,
                                                                  const uint32_t* __restrict__ bsum,
                                                                  uint32_t* __restrict__ out) {
  const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < m ? in[base + k] : 0u;
    s += v[k];
  }
  uint32_t total;
  uint32_t ex = block_excl_scan(s, &total) + bsum[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < m) out[base + k] = ex;
    ex += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[m] = bsum[blockIdx.x] + total;
}

// ---------------------------------------------------------------------------------------
// Radix sort passes.
// ---------------------------------------------------------------------------------------
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) digit_hist_kernel(const uint32_t* __restrict__ keys, size_t n,
                                                                  int shift, int tiles,
                                                                  uint32_t* __restrict__ hist) {
  __shared__ uint32_t cnt[kRadix];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * (kSortThreads * ITEMS);
#pragma unroll 4
  for (int it = 0; it < ITEMS; ++it) {
    const size_t i = base + (size_t)it * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&cnt[(keys[i] >> shift) & 0xffu], 1u);
  }
  __syncthreads();
  hist[(size_t)threadIdx.x * tiles + blockIdx.x] = cnt[threadIdx.x];
}

// Block d: exclusive scan of hist[d * tiles .. + tiles) in place; total -> digit_total[d].
__global__ void __launch_bounds__(kSortThreads) digit_scan_kernel(uint32_t* __restrict__ hist, int tiles,
                                                                  uint32_t* __restrict__ digit_total) {
  uint32_t* row = hist + (size_t)blockIdx.x * tiles;
  uint32_t carry = 0;
  for (int c0 = 0; c0 < tiles; c0 += kSortThreads) {
    const int i = c0 + threadIdx.x;
    uint32_t v = i < tiles ? row[i] : 0u;
    uint32_t total;
    uint32_t ex = block_excl_scan(v, &total);
    if (i < tiles) row[i] = ex + carry;
    carry += total;
  }
  if (threadIdx.x == 0) digit_total[blockIdx.x] = carry;
}

// Stable scatter of one tile of 256 * ITEMS keys.  Warp w owns the w-th run of 32 * ITEMS keys
// and walks it in ITEMS rounds of 32; within a round, lanes with equal digits are ranked by lane
// (match mask), and a per-warp running count per digit carries the rank across rounds.
// Warps are then ordered by an exclusive scan of the per-warp counts per digit.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads) digit_scatter_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, size_t n, int shift, int tiles, const uint32_t* __restrict__ hist,
    const uint32_t* __restrict__ digit_total) {
  __shared__ uint32_t wcnt[kSortWarps][kRadix];
  __shared__ uint32_t tile_off[kRadix];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // global offset of digit d in this tile = (sum of smaller digits) + (this digit in earlier tiles)
  {
    uint32_t total;
    uint32_t dbase = block_excl_scan(digit_total[tid], &total);
    tile_off[tid] = dbase + hist[(size_t)tid * tiles + blockIdx.x];
  }
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) wcnt[w][tid] = 0;
  __syncthreads();

  const size_t base = (size_t)blockIdx.x * (kSortThreads * ITEMS) + (size_t)warp * (32 * ITEMS);
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t key[ITEMS], val[ITEMS], rank[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)r * 32 + lane;
    const bool valid = i < n;
    key[r] = valid ? keys_in[i] : 0u;
    val[r] = valid ? vals_in[i] : 0u;
    const uint32_t dkey = valid ? ((key[r] >> shift) & 0xffu) : 0x100u;
    const uint32_t peers = __match_any_sync(0xffffffffu, dkey);
    const int leader = __ffs(peers) - 1;
    uint32_t old = 0;
    if (valid && lane == leader) {
      old = wcnt[warp][dkey];
      wcnt[warp][dkey] = old + __popc(peers);
    }
    old = __shfl_sync(0xffffffffu, old, leader);
    rank[r] = old + __popc(peers & lt_mask);
    __syncwarp();
  }
  __syncthreads();
  {  // per digit: exclusive scan over warps
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t t = wcnt[w][tid];
      wcnt[w][tid] = run;
      run += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const size_t i = base + (size_t)r * 32 + lane;
    if (i < n) {
      const uint32_t d = (key[r] >> shift) & 0xffu;
      const uint32_t pos = tile_off[d] + wcnt[warp][d] + rank[r];
      keys_out[pos] = key[r];
      vals_out[pos] = val[r];
    }
  }
}

// cell_start[c] = first sorted slot whose cell is >= c, for c = 0 .. ncells (so cell_start[ncells]
// = n), by a binary search over the sorted cells.  The position minima move as in cell_scan_kernel.
__global__ void cell_start_kernel(const uint32_t* __restrict__ cell, uint32_t n, uint32_t ncells,
                                  uint32_t* __restrict__ start, unsigned long long* minacc,
                                  unsigned long long* minout, uint32_t nmin) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t i = c; i < nmin; i += gridDim.x * blockDim.x) {
    minout[i] = minacc[i];
    minacc[i] = ~0ull;
  }
  if (c > ncells) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (__ldg(cell + mid) < c) lo = mid + 1;
    else hi = mid;
  }
  start[c] = lo;
}

// ---------------------------------------------------------------------------------------
// Counting sort.
// ---------------------------------------------------------------------------------------
constexpr int kCellScanThreads = 1024;
constexpr int kCellScanItems = kScanChunk / kCellScanThreads;
constexpr uint32_t kScanBlocks = 16384;
static_assert(kCellScanItems == 8, "two 16-byte loads per thread");

// MANY: blocks of `per_block` chunks each (all but the last), of `chunks` in all; otherwise one chunk a block.
// Every block adds up the totals of the blocks before it, so their number is kept to kScanBlocks: with one chunk a
// block a search over 4.2e9 cells takes 27.0 ms, most of it for these sums, and 8.2 with 16384 blocks (the radix
// sort 16.5); 1e9 cells 3.2 and 2.0.
template <bool MANY>
__global__ void __launch_bounds__(kCellScanThreads) cell_reduce_kernel(const uint32_t* __restrict__ count,
                                                                       uint32_t chunks, uint32_t per_block,
                                                                       uint32_t* __restrict__ chunk_total) {
  chain_begin();
  const uint32_t c0 = MANY ? blockIdx.x * per_block : blockIdx.x, c1 = MANY ? min(c0 + per_block, chunks) : c0 + 1;
  uint32_t sum = 0;
  for (uint32_t c = c0; c < c1; ++c) {
    const uint4* cp = (const uint4*)(count + (size_t)c * kScanChunk) + 2 * threadIdx.x;
    const uint4 a = cp[0], b = cp[1];
    sum += a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w;
  }
  uint32_t total;
  block_excl_scan(sum, &total);
  if (threadIdx.x == 0) chunk_total[blockIdx.x] = total;
}

// Zero rows for those of 8 consecutive cells that hold more than kBigCell (first: their first slots, just
// written; end: the slot after the last).
__device__ __noinline__ void clear_rows(uint32_t* tile_count, uint32_t tile_row, const uint32_t* first, uint32_t end) {
  for (int i = 7; i >= 0; --i) {
    const uint32_t b = first[i];
    if (end - b > kBigCell) {
      uint4* row = (uint4*)(tile_count + (size_t)(b / kBigCell) * tile_row);
      for (uint32_t w = 0; w < tile_row / 4; ++w) row[w] = make_uint4(0, 0, 0, 0);
    }
    end = b;
  }
}

// (two blocks per SM: with more than 32 registers a thread there is one, and 1e8 cells take 0.35 ms in place of 0.27)
template <bool MANY>
__global__ void __launch_bounds__(kCellScanThreads, 2) cell_scan_kernel(uint32_t* __restrict__ count, uint32_t chunks,
                                                                     uint32_t per_block,
                                                                     const uint32_t* __restrict__ chunk_total,
                                                                     uint32_t* __restrict__ start,
                                                                     uint32_t* __restrict__ tile_count,
                                                                     uint32_t tile_row, unsigned long long* minacc,
                                                                     unsigned long long* minout, uint32_t nmin) {
  __shared__ uint32_t base;
  chain_begin();
  const uint32_t tid = threadIdx.x;
  // cells of the blocks before this one
  uint32_t before = 0;
  for (uint32_t c = tid; c < blockIdx.x; c += kCellScanThreads) before += chunk_total[c];
  uint32_t total;
  block_excl_scan(before, &total);
  if (tid == 0) base = total;
  const uint32_t c0 = MANY ? blockIdx.x * per_block : blockIdx.x, c1 = MANY ? min(c0 + per_block, chunks) : c0 + 1;
  for (uint32_t c = c0; c < c1; ++c) {
    uint4* cp = (uint4*)(count + (size_t)c * kScanChunk) + 2 * tid;
    const uint4 a = cp[0], b = cp[1];
    if (a.x | a.y | a.z | a.w) cp[0] = make_uint4(0, 0, 0, 0);
    if (b.x | b.y | b.z | b.w) cp[1] = make_uint4(0, 0, 0, 0);
    const uint32_t ex = block_excl_scan(a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w, &total) + base;
    if (MANY) {
      __syncthreads();  // (base has been read)
      if (tid == 0) base += total;
    }
    uint4 o, p;
    o.x = ex;
    o.y = o.x + a.x;
    o.z = o.y + a.y;
    o.w = o.z + a.z;
    p.x = o.w + a.w;
    p.y = p.x + b.x;
    p.z = p.y + b.y;
    p.w = p.z + b.z;
    uint4* sp = (uint4*)(start + (size_t)c * kScanChunk) + 2 * tid;
    sp[0] = o;
    sp[1] = p;
    if ((a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w) > kBigCell)  // (at least their maximum)
      clear_rows(tile_count, tile_row, start + (size_t)c * kScanChunk + 8 * tid, p.w + b.w);
  }
  if (blockIdx.x == 0)
    for (uint32_t i = tid; i < nmin; i += kCellScanThreads) {
      minout[i] = minacc[i];
      minacc[i] = ~0ull;
    }
}

// The ids of cells of more than kBigCell particles, one warp per tile of consecutive ids: to their cell's
// slots in arrival order like the others; the rank of each within its cell and tile replaces its arrival rank,
// and the row of its cell gets the tile's count and the count of the tile's group of 32.  (A cell that
// large has its first slot in a block of kBigCell slots of its own, which numbers the rows.)
__device__ __noinline__ void rank_big_cells(const uint32_t* __restrict__ key, uint32_t* rank,
                                            const uint32_t* __restrict__ start, uint32_t n, uint32_t* unsorted,
                                            uint32_t* tile_count, uint32_t tile_fine, uint32_t tile_row,
                                            int tile_shift) {
  const uint32_t tile = blockIdx.x * kSortWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (tile > (n - 1) >> tile_shift) return;
  const uint32_t i0 = tile << tile_shift, len = min(1u << tile_shift, n - i0);
  uint32_t b = 0, m = 0, r = 0;  // of the id at hand: the cell's first slot and size, the arrival rank
  auto load = [&](uint32_t j) {
    m = 0;
    if (j < len) {
      const uint32_t c = key[i0 + j];
      b = start[c];
      m = start[c + 1] - b;
      r = rank[i0 + j];
    }
  };
  load(lane);
  for (uint32_t j0 = 0; j0 < len; j0 += 32) {
    const uint32_t b0 = b, r0 = r, i = i0 + j0 + lane;
    const bool big = m > kBigCell;
    load(j0 + 32 + lane);  // the next ids', while these ids' counts are read
    const unsigned peers = __match_any_sync(0xffffffffu, big ? b0 / kBigCell : 0xffffffffu);
    if (big) {
      uint32_t* row = tile_count + (size_t)(b0 / kBigCell) * tile_row;
      const int leader = __ffs(peers) - 1;
      uint32_t before = 0;
      if (lane == (uint32_t)leader) {
        before = row[tile];  // (only this warp writes the tile's counts)
        row[tile] = before + __popc(peers);
        atomicAdd(row + tile_fine + tile / 32, (uint32_t)__popc(peers));
      }
      rank[i] = __shfl_sync(peers, before, leader) + __popc(peers & ((1u << lane) - 1u));
      unsorted[b0 + r0] = i;
    }
    __syncwarp();  // the counts, for the next leaders
  }
}

// ids to their cell's slots in arrival order.
__global__ void __launch_bounds__(kSortThreads) cell_scatter_kernel(const uint32_t* __restrict__ key,
                                                                    uint32_t* rank,
                                                                    const uint32_t* __restrict__ start, uint32_t n,
                                                                    uint32_t* unsorted, uint32_t* tile_count,
                                                                    uint32_t tile_fine, uint32_t tile_row,
                                                                    int tile_shift, uint32_t* big) {
  chain_begin();
  const uint32_t i = blockIdx.x * kSortThreads + threadIdx.x;
  uint32_t c = 0, b = 0, r = 0;
  if (i < n) {
    r = *(volatile uint32_t*)(rank + i);  // (before the flag is known, not after)
    c = key[i];
    b = start[c];
  }
  const bool big_cells = *(volatile uint32_t*)big != 0;
  if (i < n && (!big_cells || start[c + 1] - b <= kBigCell)) unsorted[b + r] = i;
  if (!big_cells) return;
  rank_big_cells(key, rank, start, n, unsorted, tile_count, tile_fine, tile_row, tile_shift);
  // the block that finishes last clears the flag for the next search
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&big[1], 1u) == gridDim.x - 1) big[0] = big[1] = 0;
}

int bits_needed(uint64_t v) {
  int b = 0;
  while (v) {
    ++b;
    v >>= 1;
  }
  return b;
}

}  // namespace

size_t scan_tmp_words(size_t m) { return (m + kScanTile - 1) / kScanTile + 1; }

int launch_exclusive_scan(cudaStream_t st, const uint32_t* in, uint32_t* out, size_t m, uint32_t* tmp) {
  if (m == 0) {
    PG_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(uint32_t), st));
    return PG_OK;
  }
  const size_t nb = (m + kScanTile - 1) / kScanTile;
  scan_reduce_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(in, m, tmp);
  scan_bsum_kernel<<<1, kScanThreads, 0, st>>>(tmp, nb);
  scan_apply_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(in, m, tmp, out);
  PG_CUDA_TRY(cudaGetLastError());
  return PG_OK;
}

namespace {

constexpr int kDenseItems = 4;  // keys per thread of the radix kernels

// The sort for n particles in ncells cells, by their mean number per cell.  The more there are, the longer a
// gather thread's rank loop and the more atomics fall on one address; the radix sort's time only falls, with
// the digits.  Search and gather in us, one atomic per particle / merged per warp / radix sort, ids in
// random order and (from 256k) in cell order:
//   n    mean   random order        cell order
//   16k  593    33 / 32 / 35
//   64k  296    33 / 33 / 35
//   64k  512    40 / 38 / 36
//   256k 32     34 / 34 / 59        31 / 26 / 56
//   256k 256    55 / 56 / 58        64 / 37 / 55
//   256k 500    82 / 81 / 58       102 / 48 / 56
//   1M   16     65 / 69 / 104       54 / 52 / 80
//   1M   64     71 / 72 / 103       78 / 57 / 80
//   1M   125    83 / 83 / 100      101 / 64 / 80
//   1M   244   107 / 107 / 99      150 / 81 / 81
//   1M   579   174 / 174 / 95      265 / 131 / 81
//   4M   64    225 / 238 / 304     254 / 172 / 192
//   4M   134   245 / 255 / 302     359 / 207 / 190
//   4M   256   315 / 318 / 294     559 / 276 / 190
HashMode sort_mode(size_t n, uint64_t ncells) {
  const uint64_t mean = n / (ncells ? ncells : 1);
  if (mean >= (n >= 1000000 ? 192u : n >= 50000 ? 448u : 1024u)) return HASH_IDS;
  return mean >= 32 ? HASH_COUNT_MERGED : HASH_COUNT;
}

}  // namespace

int NbrWork::init(size_t n_, uint64_t ncells_) {
  n = n_;
  ncells = ncells_;
  mode = sort_mode(n, ncells);
  radix = mode == HASH_IDS;
  passes = (bits_needed(ncells ? ncells - 1 : 0) + 7) / 8;
  const size_t nn = n ? n : 1;
  chunks = (uint32_t)(ncells / kScanChunk + 1);
  const size_t cells = (size_t)chunks * kScanChunk;
  size_t counts = 0, tile_words = 0, nradix = 0;
  if (radix) {
    nradix = nn;
    tiles = (int)((nn + kSortThreads * kDenseItems - 1) / (kSortThreads * kDenseItems));
  } else {
    counts = cells;
    // large cells: a row of counts per tile of ids and per group of 32 tiles
    tile_shift = 10;
    while ((nn - 1) >> tile_shift >= kMaxTiles) ++tile_shift;
    tile_fine = (uint32_t)(((nn - 1) >> tile_shift) / 32 + 1) * 32;
    tile_row = tile_fine + (tile_fine / 32 + 3) / 4 * 4;
    if (nn > kBigCell) tile_words = (nn / kBigCell + 1) * tile_row;
  }
  rest_words = counts + 2;
  struct {
    uint32_t** p;
    size_t words;
  } parts[] = {{&key, nn},
               {&rank, nn},
               {&cell_start, cells},
               {&rest, rest_words},
               {&unsorted, nn - nradix},
               {&sorted_cell, nn - nradix},
               {&sorted_id, nn - nradix},
               {&chunk_total, radix ? 0 : chunks},
               {&tile_count, tile_words},
               {&key2, nradix},
               {&id2, nradix},
               {&hist, radix ? (size_t)kRadix * tiles : 0},
               {&digit_total, radix ? kRadix : 0}};
  size_t words = 0;
  for (auto& part : parts) words += (part.words + 63) / 64 * 64;  // each from a 256-byte boundary
  PG_TRY(mem.ensure(words * 4));
  uint32_t* at = mem.as<uint32_t>();
  for (auto& part : parts) {
    *part.p = at;
    at += (part.words + 63) / 64 * 64;
  }
  if (radix) {  // the buffers that the last pass writes
    sorted_cell = passes & 1 ? key2 : key;
    sorted_id = passes & 1 ? id2 : rank;
  }
  count = rest;
  big = rest + counts;
  clean = false;
  return PG_OK;
}

size_t NbrWork::bytes() const { return mem.bytes; }

NbrOrder nbr_order(const NbrWork& w) {
  NbrOrder o;
  o.unsorted = w.radix ? w.sorted_id : w.unsorted;
  o.key = w.radix ? nullptr : w.key;
  o.cell_start = w.cell_start;
  o.sorted_cell = w.sorted_cell;
  o.sorted_id = w.sorted_id;
  o.rank = w.rank;
  o.tile_count = w.tile_count;
  o.tile_fine = w.tile_fine;
  o.tile_row = w.tile_row;
  o.tile_shift = w.tile_shift;
  return o;
}

int launch_sort(cudaStream_t st, NbrWork& w, unsigned long long* minacc, unsigned long long* minout, uint32_t nmin) {
  if (w.radix) {
    uint32_t *k0 = w.key, *v0 = w.rank, *k1 = w.key2, *v1 = w.id2;
    for (int p = 0; p < w.passes; ++p) {
      digit_hist_kernel<kDenseItems><<<w.tiles, kSortThreads, 0, st>>>(k0, w.n, 8 * p, w.tiles, w.hist);
      digit_scan_kernel<<<kRadix, kSortThreads, 0, st>>>(w.hist, w.tiles, w.digit_total);
      digit_scatter_kernel<kDenseItems><<<w.tiles, kSortThreads, 0, st>>>(k0, v0, k1, v1, w.n, 8 * p, w.tiles, w.hist,
                                                                         w.digit_total);
      std::swap(k0, k1);
      std::swap(v0, v1);
    }
    cell_start_kernel<<<(unsigned)(w.ncells / 256 + 1), 256, 0, st>>>(w.sorted_cell, (uint32_t)w.n, (uint32_t)w.ncells,
                                                                     w.cell_start, minacc, minout, minacc ? nmin : 0u);
    PG_CUDA_TRY(cudaGetLastError());
    return PG_OK;
  }
  const uint32_t per_block = (w.chunks + kScanBlocks - 1) / kScanBlocks;
  const uint32_t blocks = (w.chunks + per_block - 1) / per_block;
  if (blocks > 1)
    PG_CUDA_TRY(launch_chained(st, w.n > 0, per_block > 1 ? cell_reduce_kernel<true> : cell_reduce_kernel<false>,
                               blocks, kCellScanThreads, w.count, w.chunks, per_block, w.chunk_total));
  PG_CUDA_TRY(launch_chained(st, w.n > 0 || blocks > 1,
                             per_block > 1 ? cell_scan_kernel<true> : cell_scan_kernel<false>, blocks, kCellScanThreads,
                             w.count, w.chunks, per_block, w.chunk_total, w.cell_start, w.tile_count, w.tile_row,
                             minacc, minout, minacc ? nmin : 0u));
  if (w.n)
    PG_CUDA_TRY(launch_chained(st, true, cell_scatter_kernel, (unsigned)((w.n + kSortThreads - 1) / kSortThreads),
                               kSortThreads, w.key, w.rank, w.cell_start, (uint32_t)w.n, w.unsorted, w.tile_count,
                               w.tile_fine, w.tile_row, w.tile_shift, w.big));
  PG_CUDA_TRY(cudaGetLastError());
  return PG_OK;
}

// =========================================================================================
// Cell list without device allocation (pg_cell_list_noalloc).
//
// The radix sort (digit_hist, digit_scan, digit_scatter above) needs scratch beyond its inputs and
// outputs: a second key/value buffer for the ping-pong passes, the per-tile digit histograms and
// the digit totals.  It comes from one file-scope device array, so a call allocates nothing.  Its size
// fixes the largest system it accepts (kNoAllocMaxParticles).
//
// The array is shared by every call on a device and keeps the previous call's contents.
// Nothing in it needs to start at zero: the hash writes every key, each histogram launch
// writes every bin of its tiles, the digit scan writes every total.  Calls whose work
// overlaps on the GPU (different streams, or different host threads without ordering) race
// on it.
// =========================================================================================
namespace {

constexpr size_t kNoAllocMaxParticles = 1u << 20;
constexpr size_t kNoAllocMaxTiles = (kNoAllocMaxParticles + kSortTile - 1) / kSortTile;
constexpr size_t kNoAllocKeysOff = 0;
constexpr size_t kNoAllocValsOff = kNoAllocKeysOff + 4 * kNoAllocMaxParticles;
constexpr size_t kNoAllocHistOff = kNoAllocValsOff + 4 * kNoAllocMaxParticles;
constexpr size_t kNoAllocTotalOff = kNoAllocHistOff + 4 * kRadix * kNoAllocMaxTiles;
constexpr size_t kNoAllocBytes = kNoAllocTotalOff + 4 * kRadix;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_addr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device.  The array's name in host code
// is only a host-side stand-in.  A call made outside stream capture looks the address up with
// the device current (so a cudaDeviceReset, or another context made current, is picked up) and
// keeps it per device; a call made while `st` is capturing uses the kept address of the last
// call outside capture on this device, since a lookup may have to load the module, which
// capture forbids.
int noalloc_scratch(cudaStream_t st, unsigned char** out) {
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) {
    set_error("device ordinal %d is beyond the %d devices the no-allocation cell list supports", dev,
              kNoAllocMaxDevices);
    return PG_EINVAL;
  }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
    cudaGetLastError();  // the query itself is refused while another stream captures
    cap = cudaStreamCaptureStatusActive;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (cap == cudaStreamCaptureStatusNone) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      set_error("cudaGetSymbolAddress of the cell-list scratch failed: %s", cudaGetErrorString(e));
      return PG_ECUDA;
    }
    g_noalloc_addr[dev] = p;
  } else if (!g_noalloc_addr[dev]) {
    set_error("the first no-allocation cell list call on device %d was made during stream capture; "
              "make one call on the device before capturing", dev);
    return PG_ESTATE;
  }
  *out = (unsigned char*)g_noalloc_addr[dev];
  return PG_OK;
}

// Cell index of every particle (f64 positions, id order), the same arithmetic as hash_kernel:
// c_d = clamp(floor((x_d - lo_d) * inv), 0, n_d - 1), one IEEE subtraction then one product.
struct NoAllocGrid {
  double lo[3];
  double inv;
  int n[3];
  int dim;
};

__global__ void noalloc_hash_kernel(NoAllocGrid g, const double* __restrict__ pos, uint32_t n,
                                    uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c[3] = {0, 0, 0};
  for (int d = 0; d < g.dim; ++d) {
    const double t = __dmul_rn(__dsub_rn(pos[(size_t)i * g.dim + d], g.lo[d]), g.inv);
    c[d] = !(t >= 0.0) ? 0 : (t >= (double)g.n[d] ? g.n[d] - 1 : (int)t);
  }
  keys[i] = ((uint32_t)c[2] * (uint32_t)g.n[1] + (uint32_t)c[1]) * (uint32_t)g.n[0] + (uint32_t)c[0];
  vals[i] = i;
}

// start[c] = first slot whose cell is >= c (c = 0 .. ncells), by binary search over the
// sorted cells, so every entry is written without a count buffer.
__global__ void noalloc_cell_start_kernel(const uint32_t* __restrict__ cell, uint32_t n, uint32_t ncells,
                                          uint32_t* __restrict__ start) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > ncells) return;
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (cell[mid] < c) lo = mid + 1;
    else hi = mid;
  }
  start[c] = lo;
}

}  // namespace

}  // namespace pg

extern "C" int pg_cell_list_noalloc(const double* pos, size_t n, int dim, const double domain_lo[3],
                                    const double domain_hi[3], double support, double cell_multiplier,
                                    uint32_t* sorted_cell, uint32_t* sorted_id, uint32_t* cell_start,
                                    size_t cell_start_capacity, size_t* n_cells, void* stream) {
  using namespace pg;
  clear_error();
  if (dim != 2 && dim != 3) {
    set_error("dim must be 2 or 3 (got %d)", dim);
    return PG_EINVAL;
  }
  if (!domain_lo || !domain_hi) {
    set_error("null domain bounds");
    return PG_EINVAL;
  }
  if (n > kNoAllocMaxParticles) {
    set_error("%zu particles exceed the %zu-particle limit of the no-allocation cell list", n,
              kNoAllocMaxParticles);
    return PG_EINVAL;
  }
  Grid g;
  PG_TRY(make_grid(dim, domain_lo, domain_hi, support, cell_multiplier, &g));
  const uint64_t nc = g.ncells();
  if (n_cells) *n_cells = (size_t)nc;
  if (!cell_start || cell_start_capacity < nc + 1) {
    set_error("cell_start needs %llu entries (capacity %zu)", (unsigned long long)(nc + 1), cell_start_capacity);
    return PG_EINVAL;
  }
  if (n && (!pos || !sorted_cell || !sorted_id)) {
    set_error("null position or output buffer");
    return PG_EINVAL;
  }
  unsigned char* scratch = nullptr;
  PG_TRY(noalloc_scratch((cudaStream_t)stream, &scratch));
  cudaStream_t st = (cudaStream_t)stream;
  if (n) {
    uint32_t* tmp_keys = (uint32_t*)(scratch + kNoAllocKeysOff);
    uint32_t* tmp_vals = (uint32_t*)(scratch + kNoAllocValsOff);
    uint32_t* hist = (uint32_t*)(scratch + kNoAllocHistOff);
    uint32_t* digit_total = (uint32_t*)(scratch + kNoAllocTotalOff);
    const int passes = (bits_needed(nc ? nc - 1 : 0) + 7) / 8;
    const int tiles = (int)((n + kSortTile - 1) / kSortTile);
    // Ping-pong between the scratch pair and the caller's outputs, starting on the side that
    // makes the last pass land in the outputs.
    uint32_t* kbuf[2] = {tmp_keys, sorted_cell};
    uint32_t* vbuf[2] = {tmp_vals, sorted_id};
    int cur = (passes % 2 == 0) ? 1 : 0;
    NoAllocGrid ng;
    for (int d = 0; d < 3; ++d) {
      ng.lo[d] = g.lo[d];
      ng.n[d] = g.n[d];
    }
    ng.inv = 1.0 / g.cell;
    ng.dim = dim;
    noalloc_hash_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ng, pos, (uint32_t)n, kbuf[cur], vbuf[cur]);
    for (int p = 0; p < passes; ++p) {
      const int shift = 8 * p;
      digit_hist_kernel<kSortItems><<<tiles, kSortThreads, 0, st>>>(kbuf[cur], n, shift, tiles, hist);
      digit_scan_kernel<<<kRadix, kSortThreads, 0, st>>>(hist, tiles, digit_total);
      digit_scatter_kernel<kSortItems><<<tiles, kSortThreads, 0, st>>>(kbuf[cur], vbuf[cur], kbuf[cur ^ 1],
                                                                       vbuf[cur ^ 1], n, shift, tiles, hist,
                                                                       digit_total);
      cur ^= 1;
    }
  }
  noalloc_cell_start_kernel<<<(unsigned)((nc + 1 + 255) / 256), 256, 0, st>>>(sorted_cell, (uint32_t)n, (uint32_t)nc,
                                                                             cell_start);
  PG_CUDA_TRY(cudaGetLastError());
  return PG_OK;
}
