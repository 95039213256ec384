"""Inversions in launches of many waves run 64-thread CTAs with 8 x 8 outputs a thread: the sums have the order of
the 256-thread kernel, so a simulation's bits do not depend on how many others share its handle."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import __graft_entry__ as graft

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [(6, 13), (12, 24, 33)])
def test_batched_inversions_have_the_bits_of_single_ones(sides):
    eb = graft.load_package()
    from endobeams_gb300 import scenes as S
    sdf = S.sphere_sdf()

    def net(s):
        c, p, i = S.net_on_sphere(sides[s % len(sides)], seed=s % len(sides) + 1, sdf=sdf, drop=-3e-5)
        c.nodes.ud[:] = [0.0, 0.0, -0.05]
        c.nodes.udn = c.nodes.ud.copy()
        p.tolerance_residual = 1e-4
        return c, p, i

    def run(sims):
        confs, params, inters = zip(*[net(s) for s in sims])
        eng = eb.GpuSimulations(list(confs), params[0], list(inters))
        assert all(eng.solver(k)["inverse"] > 0 for k in range(eng.n))
        dt = params[0].initial_timestep
        for frac in (1.0, 0.5):  # two factorisations
            eng.set_loads_all(eng.loads_all(dt * frac))
            k, _ = eng.step(np.full(eng.n, dt * frac))
            eng.rollback() if frac == 1.0 else eng.commit()
        out = [(int(k[s]), {f: v.copy() for f, v in eng.state(s).items()}) for s in range(eng.n)]
        eng.close()
        return out

    batch = run(range(100 * len(sides)))  # over 80 tiles an SM in the widest steps
    for s in range(len(sides)):
        (k, one), = run([s])
        for t in range(s, len(batch), len(sides)):
            assert batch[t][0] == k
            for f in ("u", "ud", "udd", "wd", "R"):
                assert np.array_equal(batch[t][1][f], one[f]), (t, f)
