"""threads_per_sim of any value up to 512 gives the bits of the library's own choice (partial warps are
rounded up); above it the engine is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(eb, scenes, threads):
    conf, p, inter = scenes.ring_drop(n_elem=37, surface="plane", height=1e-4)
    p.threads_per_sim = threads
    res = eb.run_simulations([conf], p, [inter], max_steps=2)
    return conf.nodes.un.copy(), res.ks[0], res.krylov_iterations[0]


def test_any_thread_count_gives_the_same_bits(eb, scenes):
    u0, k0, it0 = _run(eb, scenes, 0)
    for threads in (1, 31, 33, 100, 511):
        u, k, it = _run(eb, scenes, threads)
        assert (k, it) == (k0, it0) and np.array_equal(u, u0)


def test_too_many_threads_are_refused(eb, scenes):
    from endobeams_gb300 import _lib
    conf, p, inter = scenes.ring_drop(n_elem=37, surface="plane", height=1e-4)
    p.threads_per_sim = 513
    with pytest.raises(_lib.EbError, match="threads_per_sim"):
        eb.GpuSimulations([conf], p, [inter])
