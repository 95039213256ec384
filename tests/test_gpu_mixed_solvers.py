"""Simulations with a band LU and simulations with an explicit inverse in one handle: each gives what it
gives alone, whatever their order.  The condensation's lists hold the kept blocks of both; a fill that
does not tell them apart writes an inverse simulation's blocks over the next band, or past the last
one.  A 42-a-side net keeps more than 2,048 DOFs (band), a ring and a small net fewer (inverse).
Bits equal: every simulation's arithmetic is its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SDF = {}


def _scene(scenes, name):
    if name == "ring":
        return scenes.ring_drop(n_elem=64, surface="plane", height=1e-4)
    if not SDF:
        SDF[0] = scenes.sphere_sdf(n=48, h=0.8e-3)
    return scenes.net_on_sphere(int(name), seed=3, sdf=SDF[0], drop=-2e-5)


def _run(eb, scenes, names):
    built = [_scene(scenes, n) for n in names]
    p = built[0][1]
    p.tolerance_residual = 1e-4
    p.initial_timestep = 5e-5
    p.refactor_its = 8
    eng = eb.GpuSimulations([b[0] for b in built], p, [b[2] for b in built])
    kinds = [eng.solver(s) for s in range(len(names))]
    dt = np.full(len(names), p.initial_timestep)
    for _ in range(2):
        eng.set_loads_all(eng.loads_all(0.0))
        k, status = eng.step(dt)
        assert (np.asarray(status) == 0).all()
        eng.commit()
    out = [eng.state(s)["u"].copy() for s in range(len(names))]
    eng.close()
    return out, kinds


def test_band_and_inverse_simulations_share_a_handle(eb, scenes):
    alone = {n: _run(eb, scenes, [n])[0][0] for n in ("42", "23", "ring")}
    for names in (["42", "ring"], ["ring", "42"], ["23", "42", "ring", "42", "23"]):
        out, kinds = _run(eb, scenes, names)
        for n, u, k in zip(names, out, kinds):
            assert (k["band"] > 0, k["inverse"] > 0) == ((True, False) if n == "42" else (False, True)), k
            assert np.array_equal(u, alone[n]), (names, n)
