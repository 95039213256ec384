"""The network's kernels at the edges of their row tiles (16, 32 and 56 rows, chosen by the row count
against the number of SMs) and of the SM count, against the float64 oracle.

Tolerances as for the ordinary sizes: sums of at most 128 products in FP32 (forward: 1e-4 of the
largest output), then over the rows and CTAs of the batch (gradient: 2e-4 of each block's largest
entry).  A row's output does not depend on the tile: bits equal between batches of different size."""
import numpy as np
import pytest

import mlp_oracle as M

pytestmark = pytest.mark.gpu
SIZES = [1, 15, 17, 152 * 16, 152 * 16 + 1, 152 * 32, 152 * 32 + 1, 152 * 56 + 1]


@pytest.mark.parametrize("n", SIZES)
def test_tiles_match_oracle(eb, n):
    from endobeams_gb300 import warm_start as W
    rng = np.random.default_rng(n)
    p = M.init_params(3, out_gain=1.0)
    X = rng.standard_normal((n, M.NIN)).astype(np.float32)
    T = rng.standard_normal((n, M.NOUT)).astype(np.float32)
    Y, R = W.mlp_forward(p, X), M.forward(p, X)
    assert np.abs(Y - R).max() <= 1e-4 * max(1.0, np.abs(R).max())
    k = min(n, 9)
    assert np.array_equal(W.mlp_forward(p, X[-k:]), Y[-k:])
    loss, g = W.mlp_loss_grad(p, X, T)
    rl, rg = M.loss_grad(p, X, T)
    assert abs(loss - rl) <= 1e-5 * rl
    for a, b in ((M.OFF_W1, M.OFF_B1), (M.OFF_B1, M.OFF_W2), (M.OFF_W2, M.OFF_B2), (M.OFF_B2, M.OFF_W3),
                 (M.OFF_W3, M.OFF_B3), (M.OFF_B3, M.NPARAMS)):
        ref = rg[a:b]
        assert np.abs(g[a:b] - ref).max() <= 2e-4 * np.abs(ref).max(), (a, b)
