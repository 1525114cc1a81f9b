"""Double-word steps whose neighbour lists overflow: the terms of the walk that continues a full list are
added where the list's next terms would be, so a list capacity changes no bit.  Systems of the small-handle
passes (2 or 4 threads per particle) and of the general pass, both dimensions, the overlapped schedule,
and graph replay, each against the same system with lists that hold every neighbour."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu


def _lattice(n):
    return workloads.sph_lattice_3d(n=n, seed=n % 97, f64_mode=1)


def _dam(dx):
    w = workloads.dam_break_2d(dx=dx, f64_mode=1)
    w["fields"]["vel"] = np.random.default_rng(8).normal(0.0, 0.1, size=w["fields"]["vel"].shape)
    return w


CASES = [("lattice 700", lambda: _lattice(700), 5), ("lattice 5000", lambda: _lattice(5000), 40),
         ("lattice 20000", lambda: _lattice(20000), 33), ("lattice 40000", lambda: _lattice(40000), 20),
         ("lattice 40000, one entry", lambda: _lattice(40000), 1), ("dam 6518", lambda: _dam(0.02), 7),
         ("dam 39585", lambda: _dam(0.0075), 11), ("lattice 1048577", lambda: _lattice(1048577), 60)]


def _run(w, capacity, graph):
    s = ParticleSystem(make_config(**dict(w["config"], list_capacity=capacity)), w["n"])
    workloads.load_into(s, w)
    s.enable_graph(graph)
    s.step(1)
    longest = s.pair_counts().max()
    s.step(2)
    out = {k: s.get(k) for k in ("pos", "vel", "rho")}
    if not graph:
        out["acc"], out["drho"] = s.compute_rates()
    s.close()
    return out, longest


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name,make,capacity", CASES)
def test_capacity_changes_no_bit(pg, name, make, capacity, graph):
    w = make()
    ref, longest = _run(w, 0, graph)
    got, longest_cut = _run(w, capacity, graph)
    default = 64 if w["config"]["dim"] == 2 else 128
    assert capacity < longest <= default and longest_cut == longest
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k
