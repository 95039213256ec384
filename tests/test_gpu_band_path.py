"""The band LU and its sweeps on scenes that keep more DOFs than are inverted (nets of 42 and 43 a side), asserted
from the handle: staged against unstaged sweeps, two occupancy classes in one handle, tensor-core against
FP32 factors and the oracle's exact LU."""
import numpy as np
import pytest

import bridge

pytestmark = pytest.mark.gpu
L = 0.043  # size of the larger net
SDF = {}


def _scene(scenes, name):
    if name == "ring":
        return scenes.ring_drop(n_elem=64, surface="plane", height=1e-4)
    if not SDF:
        SDF[0] = scenes.sphere_sdf(n=48, h=0.8e-3)
    return scenes.net_on_sphere(int(name), seed=3, sdf=SDF[0], drop=-2e-5)


def _run(eb, scenes, names, steps=2, **params):
    built = [_scene(scenes, n) for n in names]
    p = built[0][1]
    p.tolerance_residual = 1e-4
    p.initial_timestep = 5e-5
    for k, v in params.items():
        setattr(p, k, v)
    eng = eb.GpuSimulations([b[0] for b in built], p, [b[2] for b in built])
    kinds = [eng.solver(s) for s in range(len(names))]
    ks, its = [], 0
    for _ in range(steps):
        eng.set_loads_all(eng.loads_all(0.0))
        k, status = eng.step(np.full(len(names), p.initial_timestep))
        assert (np.asarray(status) == 0).all()
        ks.append([int(x) for x in k])
        its += sum(s["krylov_iterations"] for s in eng.stats())
        eng.commit()
    out = [eng.state(s)["u"].copy() for s in range(len(names))]
    eng.close()
    return out, kinds, ks, its


@pytest.mark.parametrize("side,restart", [("42", 64), ("43", 64), ("43", 128)])
def test_staged_sweeps_give_the_bits_of_unstaged_ones(eb, scenes, side, restart):
    """restart 128: the sums' buffers leave no room beside the Hessenberg matrix, so both run unstaged or
    with four inner products a reduction."""
    a = _run(eb, scenes, [side], krylov_restart=restart)
    b = _run(eb, scenes, [side], krylov_restart=restart, stage_band=0)
    assert a[1][0]["band"] > 0 and b[1][0]["band"] == a[1][0]["band"]
    assert a[1][0]["staged"] == (restart == 64) and not b[1][0]["staged"]
    assert a[2:] == b[2:] and np.array_equal(a[0][0], b[0][0])


def test_two_occupancy_classes_of_bands(eb, scenes):
    """A wide band, a band whose staged solve fits twice on an SM, and an inverse: two launches, every
    simulation as alone."""
    p = dict(krylov_restart=16)
    alone = {n: _run(eb, scenes, [n], **p) for n in ("42", "43", "ring")}
    assert not any(a[1][0]["two_classes"] for a in alone.values())
    for names in (["42", "43", "ring"], ["ring", "43", "42", "43"]):
        out, kinds, _, _ = _run(eb, scenes, names, **p)
        for n, u, k in zip(names, out, kinds):
            assert k["two_classes"] and k["staged"] == (n != "ring") and (k["inverse"] > 0) == (n == "ring")
            assert np.array_equal(u, alone[n][0][0]), (names, n)


def test_tensor_core_band_lu_of_a_net(eb, O, scenes):
    """Every solve with fresh factors: the tensor-core and the FP32 factorisation take the oracle's steps."""
    out = {lu: _run(eb, scenes, ["43"], refactor_its=0, band_lu=lu) for lu in ("fp32", "tensor")}
    assert [out[lu][1][0]["tensor_lu"] for lu in ("fp32", "tensor")] == [False, True]
    conf, p, inter = _scene(scenes, "43")
    p.tolerance_residual = 1e-4
    p.simulation_end_time = 2 * p.initial_timestep
    m = O.OracleModel(bridge.scene_from_conf(conf, inter), bridge.params_from(p))
    rr = O.run_simulation(m)
    assert [k[0] for k in out["fp32"][2]] == [k[0] for k in out["tensor"][2]] == rr["ks"]
    assert np.abs(out["tensor"][0][0] - out["fp32"][0][0]).max() <= 1e-9 * L
    assert np.abs(out["tensor"][0][0] - m.un).max() <= 1e-6 * L
    assert out["tensor"][3] <= 1.15 * out["fp32"][3] + 2
