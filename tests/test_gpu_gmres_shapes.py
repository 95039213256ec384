"""The Krylov team's launch shape (threads per CTA, and by them the CTAs per simulation; csrc/eb_gmres.cu)
does not reach the results: sums are taken in a fixed order of chunks, rows by lanes that the plan
fixes.  A net has levels whose rows are summed by whole warps and levels that one CTA walks alone, a
stent lanes per row, a ring one CTA with its vectors in shared memory.  Bits equal, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(eb, scenes, name, threads):
    if name == "net":
        built = scenes.net_on_sphere(23, seed=3, sdf=scenes.sphere_sdf(n=48, h=0.8e-3), drop=-2e-5)
    elif name == "stent":
        built = scenes.braided_stent(wires=24, elems_per_wire=60, grid=None)
    else:
        built = scenes.ring_drop(n_elem=37, surface="plane", height=1e-4)
    p = built[1]
    p.threads_per_sim = threads
    res = eb.run_simulations([built[0]], p, [built[2]], max_steps=2)
    return built[0].nodes.un.copy(), res.ks[0], res.krylov_iterations[0]


@pytest.mark.parametrize("name", ["ring", "net", "stent"])
def test_threads_do_not_reach_the_results(eb, scenes, name):
    u0, k0, it0 = _run(eb, scenes, name, 0)
    for threads in (32, 96, 256, 512):
        u, k, it = _run(eb, scenes, name, threads)
        assert (k, it) == (k0, it0)
        assert np.array_equal(u, u0)
