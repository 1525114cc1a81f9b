"""The passes of small handles (2 or 4 threads per particle, the terms added in list order) give the bits
of the general pass (one thread per particle): a system stepped alone against the same system in a
batch too large for the small-handle passes.  Sizes at the edges of warps, blocks and of the rule
(16384 and 32768 particles double-word, 28672 and 57344 in f32), both dimensions, overflowing lists,
isolated particles, graph replay."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "rho", "mass")


def _lattice(n, seed, **cfg):
    w = workloads.sph_lattice_3d(n=n, seed=seed)
    return dict(w, config={**w["config"], "precision": 1, "f64_mode": 1, **cfg})


def _dam(n, seed, **cfg):
    """n particles of a disturbed 2D dam break, two of them at the same place and one far off."""
    w = workloads.dam_break_2d(dx=(2.0 / (0.8 * n + 400)) ** 0.5 / 1.2, precision=1, f64_mode=1)
    rng = np.random.default_rng(seed)
    f = {k: np.array(v[:n]) for k, v in w["fields"].items()}
    assert len(f["rho"]) == n
    f["vel"] = rng.normal(0.0, 0.1, size=f["vel"].shape)
    if n > 40:
        f["pos"][33] = f["pos"][7]
        f["pos"][5] = [-50.0, 80.0]
    return {"config": {**w["config"], "precision": 1, "f64_mode": 1, "n_fluid": n, **cfg}, "n": n, "fields": f}


CASES = [("lattice1", lambda: _lattice(1, 1)), ("lattice31", lambda: _lattice(31, 2)), ("lattice1003", lambda: _lattice(1003, 3)),
         ("lattice4099_half_cells", lambda: _lattice(4099, 4, cell_multiplier=0.5)),
         ("lattice16384", lambda: _lattice(16384, 5)), ("lattice16385", lambda: _lattice(16385, 6)),
         ("lattice32768", lambda: _lattice(32768, 7)),
         ("lattice3000_overflow", lambda: _lattice(3000, 8, list_capacity=20)),
         ("lattice20000_overflow", lambda: _lattice(20000, 9, list_capacity=33)),
         ("dam33", lambda: _dam(33, 10)), ("dam1500", lambda: _dam(1500, 11)), ("dam6518", lambda: _dam(6518, 12)),
         ("dam17001", lambda: _dam(17001, 13)), ("dam900_overflow", lambda: _dam(900, 14, list_capacity=6))]


F32_CASES = [c for c in CASES if "32768" not in c[0] and "17001" not in c[0]] + [
    ("lattice28673", lambda: _lattice(28673, 15)), ("lattice57344", lambda: _lattice(57344, 16)),
    ("dam30001", lambda: _dam(30001, 17))]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name,make", CASES)
def test_small_handles_give_the_bits_of_the_general_pass(pg, name, make, graph):
    _compare(make(), graph, precision=1, f64_mode=1)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name,make", F32_CASES)
def test_small_f32_handles_give_the_bits_of_the_general_pass(pg, name, make, mode):
    _compare(make(), False, precision=0, f64_mode=mode)


def _compare(w, graph, **arith):
    cfg = dict(w["config"], **arith)
    filler = _lattice(60000, 99, **arith) if cfg["dim"] == 3 else _dam(60000, 98, **arith)
    alone = ParticleSystem(make_config(**cfg), w["n"])
    both = ParticleSystem.batch([cfg, dict(filler["config"], list_capacity=cfg.get("list_capacity", 0),
                                           cell_multiplier=cfg.get("cell_multiplier", 1.0))], [w["n"], filler["n"]])
    for k in FIELDS:
        alone.set(k, np.asarray(w["fields"][k], np.float64))
        both.set(k, np.concatenate([w["fields"][k], filler["fields"][k]]).astype(np.float64))
    for s in (alone, both):
        s.enable_graph(graph)
        s.step(3)
    for k in ("pos", "vel", "rho"):
        assert np.array_equal(alone.get(k), both.get(k)[:w["n"]], equal_nan=True), k
    alone.close()
    both.close()
