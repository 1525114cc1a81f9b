// The kernels' index helpers on the host, with integer overflow reported by the compiler's sanitizer
// (run by tests/test_index_math.py):
//   rows of grids of up to 2^32 cells, those just outside included, as the walks form them
//   the slots of kernels with several threads a slot, up to 2^32 slots
#include <cstdint>
#include <cstdio>

#include "../../prestige_gb300/csrc/pg_internal.cuh"

using namespace pg;

static int bad = 0;

static void rows(int nx, int ny, int nz, uint32_t base) {
  GridK g = {};
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.cell_base = base;
  const int zs[] = {-2, -1, 0, 1, nz / 2, nz - 2, nz - 1, nz, nz + 1};
  const int ys[] = {-2, -1, 0, 1, ny / 2, ny - 2, ny - 1, ny, ny + 1};
  for (int z : zs)
    for (int y : ys) {
      const int64_t cell = (int64_t)base + ((int64_t)z * ny + y) * (int64_t)nx;
      if (row_base(g, y, z) != (uint32_t)(uint64_t)cell) {
        fprintf(stderr, "grid %d x %d x %d, row (%d, %d): %u\n", nx, ny, nz, y, z, row_base(g, y, z));
        ++bad;
      }
    }
}

template <int LANES>
static void lanes(uint32_t block) {
  for (uint64_t slot : {0ull, 1ull, 31ull, 1000000ull, (1ull << 30) - 1, 1ull << 30, (1ull << 30) + 77, 3000000001ull,
                        0xffffffefull})
    for (uint32_t sub = 0; sub < LANES; ++sub) {
      const uint64_t thread = slot * LANES + sub;
      const uint32_t b = (uint32_t)(thread / block), t = (uint32_t)(thread % block);
      if (lane_slot<LANES>(b, block, t) != slot || t % LANES != sub) {
        fprintf(stderr, "%d threads a slot, blocks of %u, slot %llu: %u\n", LANES, block, (unsigned long long)slot,
                lane_slot<LANES>(b, block, t));
        ++bad;
      }
    }
}

int main() {
  rows(10, 10, 1, 0);
  rows(1625, 1625, 1625, 0);           // 4.29e9 cells
  rows(4, 40000, 26000, 0);            // z ny alone is below 2^31, its rows are not
  rows(1, 65535, 65535, 0);            // z ny beyond 2^31
  rows(46341, 46341, 1, 0);            // 2D
  rows(1000, 1000, 1000, 3000000000u);  // a later system of a batch
  for (uint32_t block : {32u, 64u, 96u, 128u, 256u}) {
    lanes<1>(block);
    lanes<2>(block);
    lanes<4>(block);
  }
  return bad ? 1 : 0;
}
