"""The neighbour-list kernel's candidate batches at their edges: systems of a few particles, so that
rows start and end at every offset within a batch (8 or 16 slots, aligned to 4), in 2D and 3D,
cell multipliers 1 and 1/2, f64 (both modes) and f32, with coincident particles, a NaN position
and lists that fill within a batch.  The lists are integers: they must equal the oracle's."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config

pytestmark = pytest.mark.gpu


def _lists(pos, cfg, cap=0):
    n = pos.shape[0]
    s = ParticleSystem(make_config(list_capacity=cap, **cfg), n)
    s.set("pos", pos)
    s.set("vel", np.zeros_like(pos))
    s.set("rho", np.full(n, 1000.0))
    s.set("mass", np.ones(n))
    s.compute_rates()
    lengths, entries = s.pair_lists()
    _, ids, _ = s.neighbors()
    s.close()
    return lengths, entries, ids


def _oracle(oracle, pos, cfg, f64):
    dt = np.float64 if f64 else np.float32
    offs, nbr = oracle.neighbor_list(pos, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"], cfg["cell_multiplier"],
                                     f64=f64)
    x = pos.astype(dt)
    out = []
    for i in range(pos.shape[0]):
        j = nbr[offs[i]:offs[i + 1]]
        d = x[i] - x[j]
        r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
        if pos.shape[1] == 3:
            r2 = r2 + d[:, 2] * d[:, 2]
        out.append(j[r2 > 0])
    return out


@pytest.mark.parametrize("precision,mode", [(1, 0), (1, 1), (0, 0), (0, 1)])
@pytest.mark.parametrize("mult", [1.0, 0.5])
@pytest.mark.parametrize("dim", [2, 3])
def test_small_systems(pg, oracle, dim, mult, precision, mode):
    for n in (1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 31, 32, 33, 47, 65, 130):
        rng = np.random.default_rng(100 * n + dim)
        cfg = dict(model=0, dim=dim, precision=precision, f64_mode=mode, h=0.1, cell_multiplier=mult,
                   domain_lo=[0.0] * 3, domain_hi=[1.0] * 3)
        side = (n / 30.0) ** (1.0 / dim) * 0.4  # about 30 particles in a 0.4-wide region
        pos = rng.uniform(0.0, max(side, 0.15), size=(n, dim)) + 0.05
        if n > 4:
            pos[n // 2] = pos[1]  # coincident
        if precision == 0 and mode == 1:
            # f32 with fused multiply-adds shares the IEEE list test
            pos = pos.astype(np.float32).astype(np.float64)
        lengths, entries, ids = _lists(pos, cfg, cap=160)
        ref = _oracle(oracle, pos, cfg, precision == 1)
        for k in range(n):
            got = ids[entries[k, :lengths[k]]]
            assert np.array_equal(got, ref[ids[k]]), (n, k)


@pytest.mark.parametrize("mult", [1.0, 0.5])
@pytest.mark.parametrize("mode", [0, 1])
def test_lists_that_fill_within_a_batch(pg, oracle, mode, mult):
    rng = np.random.default_rng(5)
    cfg = dict(model=0, dim=3, precision=1, f64_mode=mode, h=0.1, cell_multiplier=mult, domain_lo=[0.0] * 3,
               domain_hi=[1.0] * 3)
    pos = rng.uniform(0.3, 0.6, size=(100, 3))
    ref = _oracle(oracle, pos, cfg, True)
    for cap in (1, 3, 8, 9, 17):
        lengths, entries, ids = _lists(pos, cfg, cap=cap)
        for k in range(100):
            r = ref[ids[k]]
            m = min(cap, len(r))
            assert lengths[k] == len(r)
            assert np.array_equal(ids[entries[k, :m]], r[:m])


@pytest.mark.parametrize("mode", [0, 1])
def test_nan_position_has_no_neighbours(pg, mode):
    rng = np.random.default_rng(6)
    pos = rng.uniform(0.3, 0.5, size=(40, 3))
    pos[7, 1] = np.nan
    cfg = dict(model=0, dim=3, precision=1, f64_mode=mode, h=0.1, domain_lo=[0.0] * 3, domain_hi=[1.0] * 3)
    lengths, entries, ids = _lists(pos, cfg)
    for k in range(40):
        got = ids[entries[k, :lengths[k]]]
        assert 7 not in got
        if ids[k] == 7:
            assert lengths[k] == 0


# (dim, offset of all positions, scale of positions and support): ordinary; FP32 positions that resolve
# the support poorly or not at all; squares of the support outside the FP32 range
_SCALES = [(2, 0.0, 1.0), (3, 0.0, 1.0), (3, 1e5, 1.0), (3, 1e8, 1.0), (2, 0.0, 1e-22), (3, 0.0, 1e22)]


@pytest.mark.parametrize("f64", [True, False])
@pytest.mark.parametrize("mult", [1.0, 0.5])
@pytest.mark.parametrize("dim,offset,scale", _SCALES)
def test_counts_lists_and_gather(pg, oracle, dim, offset, scale, mult, f64):
    if not f64 and (offset or scale != 1.0):
        pytest.skip("f32 systems use the IEEE FP32 test at any scale")
    for n in (1, 4, 9, 17, 33, 64, 150):
        rng = np.random.default_rng(n + dim)
        side = max(0.3, (n / 30.0) ** (1.0 / dim) * 0.4)
        pos = (rng.uniform(0.0, side, size=(n, dim)) + 0.05) * scale + offset
        if n > 4:
            pos[n - 1] = pos[2]
        h = 0.1 * scale
        lo, hi = [offset] * 3, [offset + 2.0 * scale] * 3
        cfg = dict(model=0, dim=dim, precision=1 if f64 else 0, h=h, cell_multiplier=mult, domain_lo=lo, domain_hi=hi)
        s = ParticleSystem(make_config(**cfg), n)
        s.set("pos", pos)
        src, dst = rng.normal(size=n), rng.normal(size=n)
        s.set("src", src)
        s.set("dst", dst)
        assert np.array_equal(s.count_neighbors(), oracle.neighbor_counts(pos, lo, hi, 2.0 * h, mult, f64=f64))
        offs, nbr = s.neighbor_list()
        ro, rn = oracle.neighbor_list(pos, lo, hi, 2.0 * h, mult, f64=f64)
        assert np.array_equal(offs, ro) and np.array_equal(nbr, rn)
        s.gather_sum("dst", "src")
        assert np.array_equal(s.get("dst"), oracle.gather_sum(pos, lo, hi, 2.0 * h, src, dst, mult, f64=f64))
        s.close()
