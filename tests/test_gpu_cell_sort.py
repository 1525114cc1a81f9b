"""The counting sort of the neighbour search at its edges: cells of up to and beyond the size that
the gather ranks by itself, several such cells, everything in one cell, cell counts at the edges of
the scan's chunks, shuffled ids, and searches in a row (each leaves the counters ready for the
next).  Integers: equal to the oracle's stable sort."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config

pytestmark = pytest.mark.gpu


def _check(oracle, s, pos, cfg):
    cell, ids, start = s.neighbors()
    ocell, oid, ostart = oracle.cell_list(pos, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"],
                                          cfg["cell_multiplier"], cfg["precision"] == 1)
    assert np.array_equal(start, ostart)
    assert np.array_equal(ids, oid)
    assert np.array_equal(cell, ocell[oid])


def _cfg(dim, cells, precision=1, mode=0):
    """A grid of `cells` cells of side 0.2 along x (and one cell across)."""
    side = 0.2 * (1 + 2.0 ** -20)
    return dict(model=0, dim=dim, precision=precision, f64_mode=mode, h=0.1, cell_multiplier=1.0,
                domain_lo=[0.0] * 3, domain_hi=[(cells - 0.5) * side, 0.1, 0.1])


def _in_cells(rng, counts, dim):
    """Positions with counts[c] particles in cell c, ids shuffled."""
    c = np.repeat(np.arange(len(counts)), counts)
    pos = np.full((c.size, dim), 0.05)
    pos[:, 0] = (c + rng.uniform(0.1, 0.9, size=c.size)) * 0.2 * (1 + 2.0 ** -20)
    return pos[rng.permutation(c.size)]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("counts", [(1023, 1), (1024, 3), (1025, 2), (1, 1026, 0, 2), (5000, 1500, 7, 1025, 0, 40000),
                                    (70000,), (300000, 5)])
def test_large_cells(pg, oracle, counts, dim, mode):
    rng = np.random.default_rng(len(counts) + counts[0])
    cfg = _cfg(dim, len(counts), mode=mode)
    pos = _in_cells(rng, counts, dim)
    s = ParticleSystem(make_config(**cfg), pos.shape[0])
    for _ in range(3):
        s.set("pos", pos)
        _check(oracle, s, pos, cfg)
        pos = pos[rng.permutation(pos.shape[0])]
    pos = _in_cells(rng, [pos.shape[0] // len(counts)] * len(counts), dim)  # then an even spread
    pos = np.concatenate([pos, np.full((s.n - pos.shape[0], dim), 0.01)])
    s.set("pos", pos)
    _check(oracle, s, pos, cfg)
    s.close()


@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("cells", [1, 2, 8190, 8191, 8192, 8193, 16384, 40000])
def test_scan_chunks(pg, oracle, cells, precision):
    rng = np.random.default_rng(cells)
    cfg = _cfg(2, cells, precision=precision)
    for n in (1, 31, 300, 5000):
        pos = np.stack([rng.uniform(-0.1, cells * 0.2, size=n), rng.uniform(0.0, 0.1, size=n)], 1)
        s = ParticleSystem(make_config(**cfg), n)
        for _ in range(2):
            s.set("pos", pos)
            _check(oracle, s, pos, cfg)
            pos = pos[::-1].copy()
        s.close()


def test_no_particles(pg):
    s = ParticleSystem(make_config(**_cfg(3, 5)), 0)
    _, _, start = s.neighbors()
    assert not start.any()
    s.step(2)
    s.close()
