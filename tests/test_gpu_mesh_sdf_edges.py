"""Mesh-to-SDF where the FP32 culling and sign paths could go wrong: open meshes (generalized winding
numbers of any value), needles and zero-area triangles, grids of one point, ragged bricks and flat
grids, a grid equidistant from more triangles than the candidate list holds, tiny and huge units.
Against the oracle's all-pairs FP64: the distance is the same minimum (1e-13 of the size, the bar of
the closed-mesh test); the sign where the point is not on the surface."""
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


@pytest.mark.parametrize("dims", [(1, 1, 1), (9, 5, 3), (8, 4, 4), (17, 1, 6)])
def test_open_mesh_ragged_grids(eb, dims):
    V, T = M.icosphere(2, 1.0)
    _check(eb, V, T[::2], (-0.83, -0.71, -0.62), 0.19, dims)


@pytest.mark.parametrize("unit", [1e-9, 1.0, 1e6])
def test_needles_and_zero_area_triangles(eb, unit):
    V, T = M.cube_mesh()
    V = np.concatenate([V, [[0.2, 0.2, 0.2], [0.8, 0.2, 0.2000001], [0.5, 0.2, 0.2], [0.3, 0.7, 0.4]]])
    n = len(V)
    T = np.concatenate([T, [[n - 4, n - 3, n - 2], [n - 1, n - 1, n - 1], [n - 4, n - 2, n - 2], [n - 4, n - 3, n - 1]]])
    _check(eb, unit * V, T, tuple(unit * x for x in (-0.5, -0.4, -0.3)), unit * 0.171, (13, 12, 11))


def test_single_triangle(eb):
    _check(eb, np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0.1]]), np.array([[0, 1, 2]]), (-1.0, -1.0, -1.0), 0.31, (8, 7, 9))


def test_equidistant_from_more_triangles_than_the_list_holds(eb):
    V, T = M.icosphere(4, 1.0)
    _check(eb, V, T, (-0.02, -0.02, -0.02), 0.01, (5, 5, 5))
