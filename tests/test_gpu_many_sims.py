"""More simulations in a handle than a grid's y axis has blocks (65,535): every one takes the step that it takes
alone.  Bits equal: a simulation's arithmetic does not depend on the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(eb, scenes, count):
    conf, p, _ = scenes.cantilever(n_elem=1, steps=10)
    eng = eb.GpuSimulations([conf] * count, p)
    eng.set_loads_all(eng.loads_all(p.initial_timestep))
    k, status = eng.step(np.full(count, p.initial_timestep))
    u = eng.displacements()
    eng.close()
    return np.asarray(k), np.asarray(status), np.asarray(u).reshape(count, -1)


def test_more_simulations_than_a_grids_y_axis(eb, scenes):
    k1, st1, u1 = _step(eb, scenes, 1)
    k, st, u = _step(eb, scenes, 65_600)
    assert st1[0] == 0 and np.abs(u1).max() > 0
    assert (st == 0).all() and (k == k1[0]).all() and (u == u1[0]).all()
