"""The per-entry store of the pair-once f64 kernels: its bytes per list entry (36 in the IEEE step, 124 in the
FP64 adjoint, beside 4 of the list), and partners too far apart in slot order for the distance that an
entry holds (rows of cells of more than 2^19 particles)."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu


def test_bytes_per_list_entry(pg):
    n = 6400
    w = workloads.differentiable_3d(n=n)
    used = []
    for capacity in (128, 160):
        s = ParticleSystem(make_config(**dict(w["config"], f64_mode=0, list_capacity=capacity)), n)
        workloads.load_into(s, w)
        step = s.memory_bytes()
        s.forward_checkpointed(2, 2)
        s.backward(s.get("pos") - w["target"])
        used.append((step, s.memory_bytes()))
        s.close()
    entries = 32 * n
    assert used[1][0] - used[0][0] == (4 + 36) * entries
    assert used[1][1] - used[0][1] == (4 + 36 + 4 + 124) * entries


def _strip(nx=230000, ny=6, dx=0.01):
    """A jittered 2D lattice, long in x: a row of cells (2.4 dx high) holds some 550,000 particles."""
    rng = np.random.default_rng(1)
    n = nx * ny
    i = np.arange(n)
    pos = np.stack([(i % nx + 0.5) * dx, (i // nx + 0.5) * dx], 1) + rng.uniform(-0.2 * dx, 0.2 * dx, size=(n, 2))
    f = {"pos": pos, "vel": rng.normal(0.0, 0.1, size=(n, 2)), "rho": 1000.0 * (1.0 + rng.uniform(-0.01, 0.01, size=n)),
         "mass": np.full(n, 1000.0 * dx * dx)}
    h = 1.2 * dx
    cfg = dict(model=0, dim=2, precision=1, f64_mode=0, domain_lo=[-4 * h] * 3, domain_hi=[nx * dx + 4 * h, ny * dx + 4 * h, 0.0],
               h=h, rho0=1000.0, c0=10.0, alpha=0.1, tait_B=1000.0 * 100.0 / 7.0, dt=0.25 * h / 10.0)
    return cfg, f, n


@pytest.mark.parametrize("capacity", [0, 9])
def test_far_partners_in_the_step(pg, oracle, capacity):
    cfg, f, n = _strip()
    s = ParticleSystem(make_config(**dict(cfg, list_capacity=capacity)), n)
    for k, v in f.items():
        s.set(k, v)
    s.step(1)
    if not capacity:  # there are such partners, and near ones
        lengths, entries = s.pair_lists()
        k = np.arange(0, n, 1001)
        far = [entries[i, :lengths[i]].astype(np.int64) - i for i in k]
        far = np.concatenate(far)
        assert (far >= 2 ** 19).any() and ((far > 0) & (far < 2 ** 19 - 1)).any()
    s.step(1)
    st = oracle.SphState(f["pos"], f["vel"], f["rho"], f["mass"])
    oracle.sph_run(dict(cfg, list_capacity=capacity), st, 2)
    for k in ("pos", "vel", "rho"):
        assert np.array_equal(s.get(k), getattr(st, k)), k
    s.close()


def test_far_partners_in_the_adjoint(pg):
    """The same run with x and y exchanged has near partners only."""
    cfg, f, n = _strip()
    target = f["pos"] + np.random.default_rng(2).normal(0.0, 1e-4, size=f["pos"].shape)
    out = []
    for swap in (False, True):
        o = [1, 0] if swap else [0, 1]
        c = dict(cfg, domain_hi=[cfg["domain_hi"][o[0]], cfg["domain_hi"][o[1]], 0.0])
        s = ParticleSystem(make_config(**c), n)
        for k, v in f.items():
            s.set(k, v[:, o] if v.ndim == 2 else v)
        s.forward_checkpointed(2, 2)
        da, dB, dv = s.backward(s.get("pos") - target[:, o])
        out.append((da, dB, dv[:, o]))
        s.close()
    # the sums run in another order; the recomputed states are double-word ones (1e-12)
    for a, b in zip(*out):
        assert np.abs(np.asarray(a) - np.asarray(b)).max() <= 1e-9 * np.abs(np.asarray(b)).max()
