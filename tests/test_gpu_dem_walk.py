"""The contact pass's walk over rows of cells: rows of up to 7 candidates are loaded side by side, a
particle next to a longer row (or with more than 15 survivors of the screen) walks row by row, and
the warp adds the contact terms six lanes per owner.  Random spheres of mixed radii, from nearly
free ones to crowds whose rows are shorter, longer and mixed; bit-exact with the oracle."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads
from prestige_gb300 import _native as nat

pytestmark = pytest.mark.gpu

RMAX = 0.5e-3


def _crowd(per_cell, n, seed, mult, capacity=40):
    rng = np.random.default_rng(seed)
    side = 2 * RMAX * (n / per_cell) ** (1.0 / 3.0)
    pos = rng.uniform(0.0, side, size=(n, 3))
    radius = RMAX * rng.uniform(0.2, 1.0, size=n)
    radius[0] = RMAX
    if n > 40:
        pos[30] = pos[31] + [0.0, 0.0, 1.0e-9]  # nearly coincident centres
    w = workloads.dem_compressed_lattice(nside=(2, 2, 2))
    cfg = dict(w["config"], domain_lo=[0.0] * 3, domain_hi=[side] * 3, wall_lo=[0.0] * 3, wall_hi=[side] * 3,
               cell_multiplier=mult, contact_capacity=capacity, r_max=RMAX, dt=1e-7)
    mass = 2600 * 4 / 3 * np.pi * radius ** 3
    return {"config": cfg, "n": n, "fields": {"pos": pos, "vel": rng.normal(0, 0.05, size=(n, 3)),
                                              "omega": rng.normal(0, 50.0, size=(n, 3)), "radius": radius,
                                              "mass": mass}}


def _both(oracle, w):
    s = ParticleSystem(make_config(**w["config"]), w["n"])
    workloads.load_into(s, w)
    f = w["fields"]
    return s, oracle.DemState(f["pos"], f["vel"], f["omega"], f["radius"], f["mass"], w["config"]["contact_capacity"])


@pytest.mark.parametrize("mult", [1.0, 0.5])
@pytest.mark.parametrize("per_cell,n", [(0.05, 1000), (0.5, 2049), (1.5, 2000), (2.3, 1999), (4.0, 1500), (1.0, 1),
                                        (1.0, 31), (1.0, 33)])
def test_crowds_are_bit_exact(pg, oracle, per_cell, n, mult):
    w = _crowd(per_cell, n, seed=int(100 * per_cell) + n, mult=mult)
    s, st = _both(oracle, w)
    for _ in range(3):
        s.step(1)
        c, _ = oracle.dem_run(w["config"], st, 1)
        assert c >= 0 and s.dem_contacts() == c
        for k in ("pos", "vel", "omega"):
            assert np.array_equal(s.get(k), getattr(st, k)), k
        pid, xi = s.dem_history()
        assert np.array_equal(pid.reshape(-1), st.hpid)
        assert np.array_equal(xi.reshape(-1), st.hxi)


def test_crowd_rows_cover_both_walks():
    """The crowds have particles on both sides of the line, and warps that hold both."""
    for per_cell, mixed in ((0.5, False), (1.5, True), (2.3, True)):
        w = _crowd(per_cell, 2000, seed=1, mult=1.0)
        cell = np.floor(w["fields"]["pos"] / (2 * RMAX)).astype(int)
        side = cell.max() + 1
        count = np.zeros((side + 2,) * 3, int)
        np.add.at(count, tuple((cell + 1).T), 1)
        rows = count[:-2] + count[1:-1] + count[2:]  # (x, y, z) cells: three neighbours along x
        longest = np.array([rows[c[0], c[1]:c[1] + 3, c[2]:c[2] + 3].max() for c in cell])
        assert (longest <= 7).any()
        assert (longest > 7).any() or not mixed


def test_crowd_beyond_the_history_capacity(pg, oracle):
    """More contacts than history entries: reported, and the state still the oracle's."""
    w = _crowd(1.5, 1000, seed=9, mult=1.0, capacity=3)
    s, st = _both(oracle, w)
    with pytest.raises(nat.PgError) as e:
        s.step(1)
    assert e.value.status == nat.PG_EOVERFLOW
    c, _ = oracle.dem_run(w["config"], st, 1)
    assert c == -1
    for k in ("pos", "vel", "omega"):
        assert np.array_equal(s.get(k), getattr(st, k)), k
