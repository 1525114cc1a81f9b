"""Inputs staged by pg_set_field_async directly before calls that run more than steps: the same results, bit for
bit, as with inputs set synchronously."""
import numpy as np
import pytest

from prestige_gb300 import ParticleSystem, make_config, workloads

pytestmark = pytest.mark.gpu


def _pinned(a):
    torch = pytest.importorskip("torch")
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
    t.numpy()[:] = np.asarray(a, np.float64).reshape(-1)
    return t


def _stage(s, fields, last):
    """Stages the fields, `last` last: each staging call first applies the one before."""
    keep = {k: _pinned(v) for k, v in sorted(fields.items(), key=lambda kv: kv[0] == last)}
    for k, t in keep.items():
        s.set_ptr_async(k, t.data_ptr(), t.numel())
    return keep


def _system(w, mode, graph):
    s = ParticleSystem(make_config(**dict(w["config"], precision=1, f64_mode=mode)), w["n"])
    workloads.load_into(s, w)
    s.enable_graph(graph)
    return s


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("last", ["a", "f", "mass", "pos"])
@pytest.mark.parametrize("bodies", [["f[i] += a[j]"], ["a[i] += 0.5 * a[j] * mass[j]", "f[i] = f[i] + a[i]"]])
def test_run_equations(pg, bodies, last, graph):
    w = workloads.sph_lattice_3d(n=3000, seed=1)
    rng = np.random.default_rng(2)
    old = {"a": rng.normal(size=3000), "f": rng.normal(size=3000)}
    new = {"a": rng.normal(size=3000), "f": rng.normal(size=3000), "mass": rng.uniform(1.0, 2.0, size=3000),
           "pos": w["fields"]["pos"] + rng.normal(0.0, 1e-3, size=(3000, 3))}
    out = []
    for staged in (False, True):
        s = _system(w, 0, graph)
        for k, v in old.items():
            s.set(k, v)
        if staged:
            keep = _stage(s, new, last)
        else:
            for k, v in new.items():
                s.set(k, v)
        s.run_equations(bodies)
        out.append({k: s.get(k) for k in ("a", "f", "mass", "pos")})
        s.wait_io()
        s.close()
    del keep
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("last", ["pos", "vel", "rho", "mass"])
@pytest.mark.parametrize("mode", [0, 1])
def test_forward_checkpointed(pg, mode, last):
    w = workloads.differentiable_3d(n=2000)
    rng = np.random.default_rng(3)
    new = {k: v * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, size=v.shape)) for k, v in w["fields"].items()}
    later = {k: v * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, size=v.shape)) for k, v in w["fields"].items()}
    out = []
    for staged in (False, True):
        s = _system(w, mode, False)
        if staged:
            keep = _stage(s, new, last)
        else:
            for k, v in new.items():
                s.set(k, v)
        s.forward_checkpointed(5, 2)
        out.append([s.get(k) for k in ("pos", "vel", "rho", "mass")])
        if staged:  # staged before the backward pass: taken by the call after it
            t = _pinned(later[last])
            s.set_ptr_async(last, t.data_ptr(), t.numel())
        out[-1] += [np.asarray(g) for g in s.backward(out[-1][0] - w["target"])]
        if staged:
            assert np.array_equal(s.get(last), later[last])
        s.wait_io()
        s.close()
    del keep
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_autotune_keeps_them(pg):
    w = workloads.sph_lattice_3d(n=1000, seed=4)
    s = _system(w, 1, False)
    vel = w["fields"]["vel"] + 0.5
    keep = _stage(s, {"vel": vel}, "vel")
    s.autotune(trial_steps=1)
    assert np.array_equal(s.get("vel"), vel)
    s.wait_io()
    s.close()
    del keep
