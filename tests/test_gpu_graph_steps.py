"""Steps replayed from graphs (four at a time, the rest one by one) against eager steps: the same bits for
every split of the steps, with the DEM history buffers swapped at each, and for the overlapped
schedule of large systems."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu


def _sph(n, mode):
    w = workloads.sph_lattice_3d(n=n, seed=3)
    w["config"].update(precision=1, f64_mode=mode)
    return w, ("pos", "vel", "rho")


def _dem():
    return workloads.dem_compressed_lattice(nside=(7, 7, 7)), ("pos", "vel", "omega")


CASES = [("ieee", lambda: _sph(2000, 0)), ("double_word", lambda: _sph(2000, 1)), ("dem", _dem),
         ("double_word_overlapped", lambda: _sph(1048577, 1))]


@pytest.mark.parametrize("splits", [(1, 3, 4), (5, 2, 9), (12,)])
@pytest.mark.parametrize("name,make", CASES)
def test_replayed_steps_are_the_eager_steps(pg, name, make, splits):
    w, fields = make()
    a, b = (ParticleSystem(make_config(**w["config"]), w["n"]) for _ in range(2))
    for s in (a, b):
        workloads.load_into(s, w)
    b.enable_graph(True)
    for k in splits:
        a.step(k)
        b.step(k)
        for f in fields:
            assert np.array_equal(a.get(f), b.get(f)), (f, k)
    if name == "dem":
        for x, y in zip(a.dem_history(), b.dem_history()):
            assert np.array_equal(x, y)
    a.close()
    b.close()
