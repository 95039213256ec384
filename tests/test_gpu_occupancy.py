"""More simulations than multiprocessors: the working vectors stay out of shared memory, or the reductions take four
inner products, where that lets two CTAs share an SM.  Neither changes a bit: every simulation as alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SDF = {}


def _run(eb, scenes, side, copies):
    if not SDF:
        SDF[0] = scenes.sphere_sdf(n=48, h=0.8e-3)
    built = [scenes.net_on_sphere(side, seed=6, sdf=SDF[0], drop=-2e-5) for _ in range(copies)]
    p = built[0][1]
    p.tolerance_residual = 1e-4
    eng = eb.GpuSimulations([b[0] for b in built], p, [b[2] for b in built])
    eng.set_loads_all(eng.loads_all(0.0))
    k, status = eng.step(np.full(copies, p.initial_timestep))
    assert (np.asarray(status) == 0).all()
    out = (set(int(x) for x in k), eng.state(copies - 1)["u"], eng.stats()[0]["krylov_iterations"])
    eng.close()
    return out


@pytest.mark.parametrize("side", [12, 17, 20, 21])  # vectors of 17, 35 and 48 KB; too large for shared memory
def test_shared_memory_of_a_large_batch(eb, scenes, side):
    k0, u0, its0 = _run(eb, scenes, side, 1)
    k, u, its = _run(eb, scenes, side, 160)
    assert k == k0 and its == its0 and np.array_equal(u, u0)
