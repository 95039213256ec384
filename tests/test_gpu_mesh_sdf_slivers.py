"""Mesh-to-SDF on thin triangles: the FP32 tests may discard a triangle only where their error stays far
below the margin.  Single slivers of every height in all vertex orders with points on and near them
beside other faces, small ones in a large extent (rounding to FP32 thins them further), and closed
tubes of slivers.  Against the oracle's all-pairs FP64: the same minimum, 1e-13 of the size."""
import numpy as np
import pytest

import mesh_oracle as M

pytestmark = pytest.mark.gpu


def _check(eb, V, T, origin, h, dims):
    size = max(np.abs(V).max(), h * max(dims))
    got = eb.DiscreteSignedDistanceField.from_mesh(V, np.asarray(T) + 1, origin, h, dims).values.ravel()
    ref = M.sdf_from_mesh(V, T, origin, h, dims)
    assert np.abs(np.abs(got) - np.abs(ref)).max() <= 1e-13 * size
    off = np.abs(ref) > 1e-9 * size
    assert np.array_equal(got[off] > 0, ref[off] > 0)


@pytest.mark.parametrize("ratio", [1.1e-3, 2e-3, 3e-3, 5e-3, 1e-2, 1.9e-2, 2.1e-2])
@pytest.mark.parametrize("size", [1.0, 1e-2, 1e-5])
def test_slivers_beside_other_faces(eb, ratio, size):
    """A fan of slivers of `size` of the extent, a grid through it, a second sheet just behind."""
    rng = np.random.default_rng(int(1e4 * ratio))
    V, T = [], []
    for s in range(30):
        d, e = np.linalg.qr(rng.standard_normal((3, 2)))[0].T
        o = size * 0.1 * rng.standard_normal(3)
        t = rng.random()
        tri = np.array([o, o + size * d, o + size * (t * d + ratio * e)])[rng.permutation(3)]
        T += [[len(V) + k for k in range(3)]]
        V += list(tri)
        V += list(tri + size * 4e-3 * np.cross(d, e))  # another face a little further away
        T += [[len(V) - 3, len(V) - 2, len(V) - 1]]
    V += [np.array([1.0, 1, 1]), np.array([1.0, 1, 0.9]), np.array([1.0, 0.9, 1])]  # the extent
    T += [[len(V) - 3, len(V) - 2, len(V) - 1]]
    h = 1.3 * size / 23
    _check(eb, np.array(V), np.array(T), tuple(-12 * h + 0.1 * size * rng.standard_normal(3)), h, (24, 23, 22))


@pytest.mark.parametrize("radius,length,seg", [(2e-3, 40e-3, 250), (4e-3, 40e-3, 600), (2e-3, 10e-3, 100)])
def test_tube_of_one_axial_segment(eb, radius, length, seg):
    """A closed tube whose side triangles run its whole length."""
    rng = np.random.default_rng(seg)
    a = 2 * np.pi * np.arange(seg) / seg
    r = radius * (1 + 0.02 * rng.standard_normal(seg))
    ring = np.stack([r * np.cos(a), r * np.sin(a)], 1)
    V = np.concatenate([np.c_[ring, np.zeros(seg)], np.c_[ring, np.full(seg, length)], [[0, 0, 0], [0, 0, length]]])
    i = np.arange(seg)
    j = (i + 1) % seg
    T = np.concatenate([np.stack([i, j, seg + i], 1), np.stack([j, seg + j, seg + i], 1),
                        np.stack([j, i, np.full(seg, 2 * seg)], 1), np.stack([seg + i, seg + j, np.full(seg, 2 * seg + 1)], 1)])
    h = 2.6 * radius / 23
    _check(eb, V, T, (-1.3 * radius, -1.3 * radius, 0.3 * length), h, (24, 24, 24))
