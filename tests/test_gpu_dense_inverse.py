"""The preconditioner's explicit inverse of the kept system (csrc/eb_dense.cu) on scenes whose kept
system is smaller than one 64-wide tile, ends inside a tile, spans many tiles, and (batched) has a
different size per simulation, against the oracle's exact sparse LU: every solve ends at the same
relative residual (1e-10), so the steps take the same Newton iterations and agree to 1e-9 of the
structure's size; an exact factorisation needs few GMRES iterations (FP32 rounding: at most 8 a
solve to 1e-10; a partial one needs hundreds)."""
import numpy as np
import pytest

import bridge

pytestmark = pytest.mark.gpu


def _scenes(scenes, name):
    sdf = scenes.sphere_sdf(n=48, h=0.8e-3)
    if name == "ring":
        built = [scenes.ring_drop(n_elem=37, surface="plane", height=1e-4)]
    elif name == "stent":
        built = [scenes.braided_stent(wires=24, elems_per_wire=60, grid=None)]
        built[0][1].tolerance_residual = 1e-8
        return built
    else:
        built = [scenes.net_on_sphere(s, seed=s, sdf=sdf, drop=-2e-5) for s in ((23,) if name == "net" else (5, 14, 20))]
    built[0][1].tolerance_residual = 1e-5
    return built


@pytest.mark.parametrize("name", ["ring", "net", "nets", "stent"])
def test_explicit_inverse_steps_match_the_oracle(eb, O, scenes, name):
    built = _scenes(scenes, name)
    p = built[0][1]
    res = eb.run_simulations([b[0] for b in built], p, [b[2] for b in built], max_steps=2)
    for s, b in enumerate(_scenes(scenes, name)):
        m = O.OracleModel(bridge.scene_from_conf(b[0], b[2]), bridge.params_from(p))
        rr = O.run_simulation(m, max_steps=2)
        assert res.ks[s] == rr["ks"]
        assert np.abs(built[s][0].nodes.un - m.un).max() <= 1e-9 * 0.02
        solves = res.newton_iterations[s] + 2
        assert res.krylov_iterations[s] <= 8 * solves * (1 if p.precision == "fp64" else 3)
