"""Element launches of many waves (a thread per element) give the bits of cooperative ones (the same simulation
alone): forces, energies' sums and states, with and without damping, at the rotations of a stent and of nets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SDF = {}


def _scene(scenes, name, damping):
    if name == "stent":
        c = scenes.braided_stent(wires=16, elems_per_wire=40, grid=None)
    else:
        if not SDF:
            SDF[0] = scenes.sphere_sdf(n=48, h=0.8e-3)
        c = scenes.net_on_sphere(20, seed=3, sdf=SDF[0], drop=-2e-5)
    c[0].beams.damping[:] = damping
    rng = np.random.default_rng(1)
    c[0].nodes.ud[:] = 0.05 * rng.standard_normal(c[0].nodes.ud.shape)
    c[0].nodes.udn = c[0].nodes.ud.copy()
    return c


def _run(eb, scenes, name, damping, copies):
    built = [_scene(scenes, name, damping) for _ in range(copies)]
    p = built[0][1]
    p.tolerance_residual, p.max_iterations = 1e-4, 3
    eng = eb.GpuSimulations([b[0] for b in built], p, [b[2] for b in built])
    k, status = eng.step(np.full(copies, p.initial_timestep))
    out = []
    for s in range(0, copies, max(1, copies - 1)):
        out.append((int(k[s]), eng.state(s), eng.forces(s)))
    eng.close()
    return out


@pytest.mark.parametrize("name,damping,elements", [("net", 0.0, 760), ("net", 20.0, 760), ("stent", 5.0, 640)])
def test_a_thread_per_element_gives_the_same_bits(eb, scenes, name, damping, elements):
    (k0, s0, f0), = _run(eb, scenes, name, damping, 1)
    copies = 448 * 152 // elements + 1
    for k, s, f in _run(eb, scenes, name, damping, copies):
        assert k == k0 and all(np.array_equal(s[x], s0[x]) for x in s0)
        assert all(np.array_equal(f[x], f0[x]) for x in f0)
