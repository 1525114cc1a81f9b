"""Neighbour searches at scales whose squared support lies near the ends of the FP32 range: the pair lists of
the SPH passes (both f64 modes and f32) and, for f32 systems, counts, CSR lists and the gather at offsets and
scales.  Integers: equal to the oracle's."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config

pytestmark = pytest.mark.gpu


def _positions(n, dim, scale, offset=0.0):
    rng = np.random.default_rng(10 * n + dim)
    side = max(0.3, (n / 30.0) ** (1.0 / dim) * 0.4)
    return (rng.uniform(0.0, side, size=(n, dim)) + 0.05) * scale + offset


def _config(dim, scale, mult, offset=0.0, **kw):
    return dict(model=0, dim=dim, h=0.1 * scale, cell_multiplier=mult, domain_lo=[offset] * 3,
                domain_hi=[offset + 2.0 * scale] * 3, **kw)


def _neighbours(oracle, pos, cfg, f64):
    """Per particle the neighbours under the oracle's test, coincident ones left out."""
    offs, nbr = oracle.neighbor_list(pos, cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"], cfg["cell_multiplier"],
                                     f64=f64)
    x = pos.astype(np.float64 if f64 else np.float32)
    out = []
    with np.errstate(over="ignore", under="ignore"):
        for i in range(pos.shape[0]):
            j = nbr[offs[i]:offs[i + 1]]
            d = x[i] - x[j]
            r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]
            if pos.shape[1] == 3:
                r2 = r2 + d[:, 2] * d[:, 2]
            out.append(j[r2 > 0])
    return out


# (2h)^2 is 2.3e38 (twice it overflows), 1.6e37, 4e-36, 4e-38
@pytest.mark.parametrize("scale", [7.5e19, 2e19, 1e-17, 1e-18])
@pytest.mark.parametrize("mult", [1.0, 0.5])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("precision,mode", [(1, 0), (1, 1), (0, 0)])
def test_pair_lists(pg, oracle, precision, mode, dim, mult, scale):
    cfg = _config(dim, scale, mult, precision=precision, f64_mode=mode, list_capacity=160)
    for n in (2, 9, 33, 150):
        pos = _positions(n, dim, scale)
        s = ParticleSystem(make_config(**cfg), n)
        s.set("pos", pos)
        s.set("vel", np.zeros_like(pos))
        s.set("rho", np.full(n, 1000.0))
        s.set("mass", np.ones(n))
        s.compute_rates()
        lengths, entries = s.pair_lists()
        _, ids, _ = s.neighbors()
        s.close()
        ref = _neighbours(oracle, pos, cfg, precision == 1)
        for k in range(n):
            assert np.array_equal(ids[entries[k, :lengths[k]]], ref[ids[k]]), (n, k)


@pytest.mark.parametrize("mult", [1.0, 0.5])
@pytest.mark.parametrize("dim,offset,scale", [(3, 1e3, 1.0), (2, 1e5, 1.0), (3, 0.0, 7.5e19), (2, 0.0, 1e-18),
                                              (3, 0.0, 1e-22)])
def test_f32_counts_lists_and_gather(pg, oracle, dim, offset, scale, mult):
    cfg = _config(dim, scale, mult, offset, precision=0)
    lo, hi, sup = cfg["domain_lo"], cfg["domain_hi"], 2.0 * cfg["h"]
    for n in (1, 17, 150):
        pos = _positions(n, dim, scale, offset)
        rng = np.random.default_rng(n)
        src, dst = rng.normal(size=n), rng.normal(size=n)
        s = ParticleSystem(make_config(**cfg), n)
        s.set("pos", pos)
        s.set("src", src)
        s.set("dst", dst)
        assert np.array_equal(s.count_neighbors(), oracle.neighbor_counts(pos, lo, hi, sup, mult, f64=False))
        offs, nbr = s.neighbor_list()
        ro, rn = oracle.neighbor_list(pos, lo, hi, sup, mult, f64=False)
        assert np.array_equal(offs, ro) and np.array_equal(nbr, rn)
        s.gather_sum("dst", "src")
        assert np.array_equal(s.get("dst"), oracle.gather_sum(pos, lo, hi, sup, src, dst, mult, f64=False))
        s.close()
