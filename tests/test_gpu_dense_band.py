"""Kept systems that are narrow bands (nets and wires that are inverted as they are or after one level): the inversion
leaves out the blocks that are still zero, and its result is still an exact preconditioner (at most 8 iterations a
solve to 1e-10, the oracle's Newton iterations, positions within 1e-9 of the structure)."""
import numpy as np
import pytest

import bridge

pytestmark = pytest.mark.gpu


def _scene(scenes, name):
    if name == "cantilever":
        c = scenes.cantilever(n_elem=32)
        c[1].tolerance_residual = 1e-5
        return c, 0.1
    c = scenes.net_on_sphere(12 if name == "net12" else 16, seed=4, sdf=scenes.sphere_sdf(n=48, h=0.8e-3), drop=-2e-5)
    c[1].tolerance_residual = 1e-5
    return c, 0.016


@pytest.mark.parametrize("name", ["cantilever", "net12", "net16"])
def test_inverse_of_a_narrow_band(eb, O, scenes, name):
    (conf, p, inter), L = _scene(scenes, name)
    res = eb.run_simulations([conf], p, [inter], max_steps=2)
    (c2, p2, i2), _ = _scene(scenes, name)
    m = O.OracleModel(bridge.scene_from_conf(c2, i2), bridge.params_from(p2))
    rr = O.run_simulation(m, max_steps=2)
    assert res.ks[0] == rr["ks"]
    assert np.abs(conf.nodes.un - m.un).max() <= 1e-9 * L
    assert res.krylov_iterations[0] <= 8 * (res.newton_iterations[0] + 2)
