"""Neighbour searches over grids of many cells: the cell table of grids beyond the size where a block of the scan
takes several chunks of cells (1.3e8), equal to the oracle's, and a search's time, which grows with the
number of cells and not with its square (34 GB for the largest)."""
import time

import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config

pytestmark = pytest.mark.gpu

SIDE = 0.2 * (1 + 2.0 ** -20)


def _system(nx, ny, n, seed):
    cfg = dict(model=0, dim=2, precision=1, h=0.1, cell_multiplier=1.0, domain_lo=[0.0] * 3,
               domain_hi=[(nx - 0.5) * SIDE, (ny - 0.5) * SIDE, 0.1], list_capacity=1)
    pos = np.random.default_rng(seed).uniform(0.0, 1.0, size=(n, 2)) * [nx * SIDE, ny * SIDE]
    s = ParticleSystem(make_config(**cfg), n)
    s.set("pos", pos)
    return s, cfg, pos


# one chunk of 8192 entries a block up to 16384 chunks; two and three chunks a block, the last block short
@pytest.mark.parametrize("nx,ny", [(16384, 8191), (16384, 8192), (20000, 13000), (20000, 13430)])
def test_cell_table(pg, oracle, nx, ny):
    s, cfg, pos = _system(nx, ny, 3000, nx + ny)
    assert s.num_cells() == nx * ny
    for _ in range(2):
        cell, ids, start = s.neighbors()
        ocell, oid, ostart = oracle.cell_list(pos, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"], 1.0, True)
        assert np.array_equal(ids, oid)
        assert np.array_equal(cell, ocell[oid])
        assert np.array_equal(start, ostart)
        pos = pos[::-1].copy()
        s.set("pos", pos)
    s.close()


def test_time_grows_with_the_cells(pg):
    def search(nx, ny):
        s, _, _ = _system(nx, ny, 1000, 1)
        best = 1e9
        for _ in range(5):
            t0 = time.perf_counter()
            s.build_neighbors()
            best = min(best, time.perf_counter() - t0)
        s.close()
        return best

    small, large = search(32500, 32300), search(65000, 64600)  # 1.05e9 and 4.2e9 cells
    assert large < 6.0 * small, (small, large)
