"""Cells of more than 1,024 particles.  In mostly empty grids their order comes from counts per tile of
consecutive ids (1,024 ids, more from 2^20 particles on); grids that hold many particles per cell on average
take the radix sort.  Sizes around that number, many such cells at once beside small ones, ids in cell
order, reversed and shuffled, several tile sizes, grids on both sides of the rule, batches, and steps;
integers equal to the oracle's stable sort.  And their cost: near that of any other search."""
import time

import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu

SIDE = 0.2 * (1 + 2.0 ** -20)


def _cfg(cells, **kw):
    """A row of `cells` cells along x."""
    return dict(dict(model=0, dim=2, precision=1, h=0.1, cell_multiplier=1.0, domain_lo=[0.0] * 3,
                     domain_hi=[(cells - 0.5) * SIDE, 0.1, 0.1], list_capacity=1), **kw)


def _positions(counts, rng, order):
    c = np.repeat(np.arange(len(counts)), counts)
    pos = np.full((c.size, 2), 0.05)
    pos[:, 0] = (c + rng.uniform(0.1, 0.9, size=c.size)) * SIDE
    return {"sorted": pos, "reversed": pos[::-1].copy(), "shuffled": pos[rng.permutation(c.size)]}[order]


def _check(oracle, s, pos, cfg):
    cell, ids, start = s.neighbors()
    ocell, oid, ostart = oracle.cell_list(pos, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"],
                                          cfg["cell_multiplier"], True)
    assert np.array_equal(start, ostart)
    assert np.array_equal(ids, oid)
    assert np.array_equal(cell, ocell[oid])


def _counts(kind, rng):
    if kind == "around 1024":
        return rng.integers(1000, 1050, size=300)
    if kind == "exactly":
        return np.array([1024, 1025, 0, 1024, 1026, 1025, 33, 32, 31, 1])
    if kind == "mixed":
        return np.where(rng.random(2000) < 0.05, rng.integers(1025, 6000, size=2000), rng.integers(0, 60, size=2000))
    if kind == "few in many":  # one and a half million cells (an extra scan of several chunks)
        c = np.zeros(1500000, int)
        c[[0, 5, 8191, 8192, 700000, 1499999]] = (1025, 70000, 1024, 2000, 100001, 1030)
        return c
    if kind == "merged":  # between 32 particles a cell and the radix sort, on average
        return np.concatenate([rng.integers(0, 300, size=800), [1025, 3000, 1024]])
    return np.array({"one": [200000], "tiles of 2048": [3, 1100000, 5, 1025], "tiles of 4096": [1500000, 2, 700000]}[kind])


@pytest.mark.parametrize("order", ["shuffled", "sorted", "reversed"])
@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("kind", ["exactly", "around 1024", "mixed", "merged", "few in many", "one", "tiles of 2048",
                                  "tiles of 4096"])
def test_order(pg, oracle, kind, empty, order):
    rng = np.random.default_rng(len(kind))
    counts = _counts(kind, rng)
    if empty:  # empty cells behind the last one, so that the mean is low
        counts = np.concatenate([counts, np.zeros(counts.sum() // 20, int)])
    cfg = _cfg(len(counts))
    pos = _positions(counts, rng, order)
    s = ParticleSystem(make_config(**cfg), pos.shape[0])
    for _ in range(2):  # the second search on what the first one left
        s.set("pos", pos)
        _check(oracle, s, pos, cfg)
        pos = np.roll(pos, 12345, axis=0)
    spread = pos.copy()  # then a search without such cells, then the first again
    spread[:, 0] = rng.uniform(0.0, len(counts) * SIDE, size=spread.shape[0])
    for p in (spread, pos):
        s.set("pos", p)
        _check(oracle, s, p, cfg)
    s.close()


@pytest.mark.parametrize("scale", [1, 10])  # counted tiles, radix sort
@pytest.mark.parametrize("mode", [0, 1])
def test_batch(pg, oracle, mode, scale):
    """Systems with and without large cells in one handle: each as in a handle of its own."""
    rng = np.random.default_rng(5)
    counts = [scale * np.array(c) for c in ([1500, 3, 2000], [20, 20, 20], [0, 5000, 1025, 1])]
    cfgs = [_cfg(len(c), f64_mode=mode) for c in counts]
    pos = [_positions(c, rng, "shuffled") for c in counts]
    s = ParticleSystem.batch(cfgs, [p.shape[0] for p in pos])
    s.set("pos", np.concatenate(pos))
    cell, ids, start = s.neighbors()
    assert (s.info()["sort_passes"] > 0) == (scale == 10)
    first = base = 0
    for p, cfg in zip(pos, cfgs):
        ocell, oid, ostart = oracle.cell_list(p, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"], 1.0, True)
        n = p.shape[0]
        assert np.array_equal(ids[first:first + n], oid + first)
        assert np.array_equal(cell[first:first + n], ocell[oid] + base)
        assert np.array_equal(start[base:base + len(ostart)], ostart + first)
        first += n
        base += len(ostart) - 1
    s.close()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n,mult", [(20000, 5.0), (60000, 4.0), (1048577, 3.0)])
@pytest.mark.parametrize("mode", [0, 1])
def test_steps(pg, mode, n, mult, graph):
    """A lattice in large cells (counted tiles, radix sort; beyond 1M particles on the overlapped schedule) against
    the same one in ordinary cells."""
    w = workloads.sph_lattice_3d(n=n, seed=11, f64_mode=mode)
    out = []
    for m in (mult, 1.0):
        s = ParticleSystem(make_config(**dict(w["config"], cell_multiplier=m)), w["n"])
        workloads.load_into(s, w)
        if m > 1.0:
            _, _, start = s.neighbors()
            assert np.diff(start.astype(np.int64)).max() > (1024 if n < 1000000 else 400)
            assert (s.info()["sort_passes"] > 0) == (n > 20000)
        s.enable_graph(graph)
        s.step(5)
        out.append([s.get(k) for k in ("pos", "vel", "rho")])
        s.close()
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()


@pytest.mark.parametrize("mode", [0, 1])
def test_batch_steps(pg, mode):
    """Three lattices in one handle (radix sort, a position minimum per system) and each alone (counted tiles):
    the same bits."""
    ws = [workloads.sph_lattice_3d(n=n, seed=n, f64_mode=mode, cell_multiplier=5.0) for n in (19000, 20000, 21000)]
    for i, w in enumerate(ws):  # apart from one another, so that the minima differ
        w["fields"]["pos"] += 10.0 * i
        for k in ("domain_lo", "domain_hi"):
            w["config"][k] = [x + 10.0 * i for x in w["config"][k]]
    both = ParticleSystem.batch([w["config"] for w in ws], [w["n"] for w in ws])
    assert both.info()["sort_passes"] > 0
    for k in ("pos", "vel", "rho", "mass"):
        both.set(k, np.concatenate([w["fields"][k] for w in ws]))
    both.step(3)
    first = 0
    for w in ws:
        s = ParticleSystem(make_config(**w["config"]), w["n"])
        assert s.info()["sort_passes"] == 0
        workloads.load_into(s, w)
        s.step(3)
        for k in ("pos", "vel", "rho"):
            assert np.array_equal(both.get(k)[first:first + w["n"]], s.get(k)), k
        first += w["n"]
        s.close()
    both.close()


def test_cost(pg):
    """Some milliseconds where one block sorts such cells; here near an ordinary search's time."""
    rng = np.random.default_rng(6)
    n = 1000000

    def search(cells, empty):
        s = ParticleSystem(make_config(**_cfg(cells + empty)), n)
        s.set("pos", _positions(rng.multinomial(n, [1.0 / cells] * cells), rng, "shuffled"))
        best = 1e9
        for _ in range(10):
            t0 = time.perf_counter()
            s.build_neighbors()
            best = min(best, time.perf_counter() - t0)
        s.close()
        return best

    ordinary = search(50000, 0)  # about 0.06 ms; one block would take 7 to 10
    for cells in (800, 100, 10):
        for empty in (0, 50000):
            assert search(cells, empty) < 20.0 * ordinary, (cells, empty)


# the means at which the sort changes (sort_mode in pg_sort.cu), with cells enough for 0, 1 and 2 radix digits
@pytest.mark.parametrize("n,cells", [(1023, 1), (1024, 1), (49999, 49), (49999, 48), (50000, 112), (50000, 111),
                                     (999999, 5208), (1000000, 5209), (1000000, 5208), (1000, 32), (1000, 31),
                                     (120000, 257)])
@pytest.mark.parametrize("precision,mode", [(1, 0), (1, 1), (0, 0)])
def test_edges_of_the_rule(pg, oracle, n, cells, precision, mode):
    rng = np.random.default_rng(n + cells)
    cfg = _cfg(cells, precision=precision, f64_mode=mode)
    s = ParticleSystem(make_config(**cfg), n)
    assert (s.info()["sort_passes"] > 0) == (cells > 1 and n // cells >= (192 if n >= 1000000 else
                                                                         448 if n >= 50000 else 1024))
    for _ in range(2):
        pos = _positions(rng.multinomial(n, [1.0 / cells] * cells), rng, "shuffled")
        s.set("pos", pos)
        cell, ids, start = s.neighbors()
        ocell, oid, ostart = oracle.cell_list(pos, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"], 1.0, precision == 1)
        assert np.array_equal(start, ostart) and np.array_equal(ids, oid) and np.array_equal(cell, ocell[oid])
    s.close()
