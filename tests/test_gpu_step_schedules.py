"""Steps in a row, eager and replayed from graphs of one and four, where the schedule differs: the overlapped
IEEE step of large systems (lists on a second stream, the last kernel chained to the next step's first),
f32 handles and batches; the IEEE ones against the oracle.  And the pair-once IEEE kernels in small
systems with lists cut short (pairs held by one list only, continued walks)."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "rho")


def _oracle_run(oracle, cfg, f, steps):
    st = oracle.SphState(f["pos"], f["vel"], f["rho"], f["mass"])
    oracle.sph_run(cfg, st, steps)
    return st


def test_overlapped_ieee_steps_in_a_row(pg, oracle):
    w = workloads.sph_lattice_3d(n=1048577, seed=3, precision=1, f64_mode=0)
    st = _oracle_run(oracle, w["config"], w["fields"], 5)
    for graph in (False, True):
        s = ParticleSystem(make_config(**w["config"]), w["n"])
        workloads.load_into(s, w)
        assert s.info()["overlap_split"] > 0
        s.enable_graph(graph)
        s.step(5)
        for k in FIELDS:
            assert np.array_equal(s.get(k), getattr(st, k)), (k, graph)
        s.close()


@pytest.mark.parametrize("n,mode", [(3000, 0), (3000, 1), (70000, 0)])
def test_f32_replays(pg, n, mode):
    w = workloads.sph_lattice_3d(n=n, seed=5, precision=0, f64_mode=mode)
    a, b = (ParticleSystem(make_config(**w["config"]), n) for _ in range(2))
    for s in (a, b):
        workloads.load_into(s, w)
    b.enable_graph(True)
    for k in (1, 4, 6):
        a.step(k)
        b.step(k)
        for f in FIELDS:
            assert np.array_equal(a.get(f), b.get(f)), (f, k)
    a.close()
    b.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_batch_replays(pg, oracle, mode):
    ws = workloads.batched_dam_breaks(n_systems=6, nmin=300, nmax=3000, f64_mode=mode)
    counts = [w["n"] for w in ws]
    a, b = (ParticleSystem.batch([w["config"] for w in ws], counts) for _ in range(2))
    for s in (a, b):
        for k in FIELDS + ("mass",):
            s.set(k, np.concatenate([np.asarray(w["fields"][k]) for w in ws]))
    b.enable_graph(True)
    for k in (3, 6):
        a.step(k)
        b.step(k)
        for f in FIELDS:
            assert np.array_equal(a.get(f), b.get(f)), (f, k)
    if mode == 0:
        first = 0
        for w in ws:
            st = _oracle_run(oracle, w["config"], w["fields"], 9)
            for f in FIELDS:
                assert np.array_equal(a.get(f)[first:first + w["n"]], getattr(st, f)), f
            first += w["n"]
    a.close()
    b.close()


@pytest.mark.parametrize("capacity", [1, 7, 30, 0])
@pytest.mark.parametrize("name", ["lattice 31", "lattice 700", "lattice 9000", "dam 1418"])
def test_small_ieee_systems_with_cut_lists(pg, oracle, name, capacity):
    n = int(name.split()[1])
    w = workloads.dam_break_2d(dx=0.05) if name.startswith("dam") else workloads.sph_lattice_3d(n=n, seed=n)
    assert w["n"] == n
    f = w["fields"]
    f["vel"] = np.random.default_rng(n).normal(0.0, 0.1, size=f["vel"].shape)
    cfg = dict(w["config"], precision=1, f64_mode=0, list_capacity=capacity)
    s = ParticleSystem(make_config(**cfg), n)
    workloads.load_into(s, w)
    s.step(3)
    st = _oracle_run(oracle, cfg, f, 3)
    for k in FIELDS:
        assert np.array_equal(s.get(k), getattr(st, k)), k
    s.close()
