"""The launch count of pg_timing: steps replayed from a graph count the kernels that the same steps count when
they are launched one by one, in every mode, for the overlapped schedules of large systems too."""
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu


def _sph(n, precision, mode):
    w = workloads.sph_lattice_3d(n=n, seed=3, precision=precision, f64_mode=mode)
    return w


# kernels of a step beyond the neighbour search's (3, or 4 for more than 8191 cells)
CASES = [("ieee", lambda: _sph(2000, 1, 0), 3 + 6), ("double word", lambda: _sph(2000, 1, 1), 3 + 4),
         ("f32", lambda: _sph(2000, 0, 0), 3 + 4), ("dem", lambda: workloads.dem_compressed_lattice(nside=(7, 7, 7)), 3 + 2),
         ("ieee overlapped", lambda: _sph(1048577, 1, 0), 4 + 8),
         ("double word overlapped", lambda: _sph(1048577, 1, 1), 4 + 6)]


@pytest.mark.parametrize("name,make,per_step", CASES)
def test_replayed_steps_count_their_kernels(pg, name, make, per_step):
    w = make()
    s = ParticleSystem(make_config(**w["config"]), w["n"])
    workloads.load_into(s, w)
    for graph in (False, True):
        s.enable_graph(graph)
        for steps in (1, 3, 4, 9):
            s.timing_enable(False)  # sets the count to zero
            s.step(steps)
            assert s.timing_read()["launches"] == steps * per_step, (graph, steps)
    s.close()
