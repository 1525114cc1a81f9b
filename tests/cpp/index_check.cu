// The kernels' index helpers on the host, with integer overflow reported by the compiler's sanitizer
// (run by tests/test_index_math.py): rows of grids of up to 2^32 cells, those just outside included, as
// the walks form them.
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

int main() {
  rows(10, 10, 1, 0);
  rows(1625, 1625, 1625, 0);           // 4.29e9 cells
  rows(4, 40000, 26000, 0);            // z ny alone is below 2^31, its rows are not
  rows(1, 65535, 65535, 0);            // z ny beyond 2^31
  rows(46341, 46341, 1, 0);            // 2D
  rows(1000, 1000, 1000, 3000000000u);  // a later system of a batch
  return bad ? 1 : 0;
}
