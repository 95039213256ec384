"""The network's sums have one order (csrc/eb_mlp.cu): an output adds its products in increasing k from
the bias, a gradient adds rows tile by tile (32 rows, a CTA's tiles are c, c + CTAs, ...) and then the
CTAs' partials in order.  With W2 = 0 the hidden activations are one vector that forward calls can
read back exactly, so those sums are formed here in the same order, each product and addition rounded
once as FP32 fma does.  Bits equal, no tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

O3 = 48 * 128 + 128 + 128 * 128 + 128  # offset of W3
f32 = np.float32


def _fma(a, b, c):  # one rounding to FP32 (the products are exact in long double, the sums to its precision)
    return (np.longdouble(a) * np.longdouble(b) + np.longdouble(c)).astype(f32)


def _network(W, rng):
    """Parameters with W2 = 0 and W3 = 0, and the hidden activations h2 of every row, read back one by one."""
    p = W.init_params(5, out_gain=1.0).astype(f32)
    p[48 * 128 + 128:O3 - 128] = 0
    p[O3 - 128:O3] = rng.standard_normal(128)
    p[O3:] = 0
    h = np.zeros(128, f32)
    for k0 in range(0, 128, 6):
        q = p.copy()
        for o in range(min(6, 128 - k0)):
            q[O3 + (k0 + o) * 6 + o] = 1
        h[k0:k0 + 6] = W.mlp_forward(q, np.zeros((1, 48), f32))[0][:128 - k0]
    return p, h


@pytest.mark.parametrize("n", [1, 17, 33, 2433, 4865, 9761])
def test_outputs_and_gradients_add_in_one_order(eb, n):
    from endobeams_gb300 import warm_start as W
    rng = np.random.default_rng(n)
    p, h = _network(W, rng)
    w3 = torch.from_numpy(rng.standard_normal((128, 6)).astype(f32)).bfloat16().float().numpy()
    b3 = rng.standard_normal(6).astype(f32)
    p[O3:O3 + 768], p[O3 + 768:] = w3.ravel(), b3
    X = rng.standard_normal((n, 48)).astype(f32)
    y = b3.copy()
    for k in range(128):
        y = _fma(h[k], w3[k], y)
    assert np.array_equal(W.mlp_forward(p, X), np.broadcast_to(y, (n, 6)))
    T = rng.standard_normal((n, 6)).astype(f32)
    T[rng.random(n) < 0.1] = np.nan
    loss, g = W.mlp_loss_grad(p, X, T)
    d = np.where(np.isnan(T), f32(0), y - T)
    assert abs(loss - (d.astype(float) ** 2).mean()) <= 1e-12 * loss
    dy = d * (f32(2) / f32(n * 6.0))
    tiles = -(-n // 32)
    ctas = min(tiles, torch.cuda.get_device_properties(0).multi_processor_count)
    dy = np.concatenate([dy, np.zeros((tiles * 32 - n, 6), f32)]).reshape(tiles, 32, 6)
    gw, gb = np.zeros((128, 6), f32), np.zeros(6, f32)
    for c in range(ctas):
        pw, pb = np.zeros((128, 6), f32), np.zeros(6, f32)
        for row in dy[c::ctas].reshape(-1, 6):
            pw, pb = _fma(h[:, None], row, pw), pb + row
        gw, gb = gw + pw, gb + pb
    assert np.array_equal(g[O3:O3 + 768].reshape(128, 6), gw)
    assert np.array_equal(g[O3 + 768:], gb)
