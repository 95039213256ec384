"""The condensation plan in front of the band LU (csrc/eb_cond_plan.hpp): on graphs of every
shape the scenes and callers can have, the planned elimination, walked in FP64 on the host with
the kernels' operations, solves the whole system (the general path: no elimination, one dense
solve) to FP64 rounding: 1e-12 of the right-hand side for block diagonally dominant matrices."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    so = str(tmp_path_factory.mktemp("cond") / "cond_host.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", os.path.join(HERE, "host", "cond_host.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    lib.host_cond_residual.restype = ctypes.c_double
    return lib


def _grid(a, b):
    i = np.arange(a * b).reshape(a, b)
    return a * b, np.concatenate([np.stack([i[:-1].ravel(), i[1:].ravel()], 1),
                                  np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)])


def _graphs():
    rng = np.random.default_rng(3)
    path = lambda n: np.stack([np.arange(n - 1), np.arange(1, n)], 1)
    yield "one node", 1, np.zeros((0, 2), int)
    yield "two nodes", 2, path(2)
    yield "no edges", 5, np.zeros((0, 2), int)
    yield "path 21", 21, path(21)
    perm = rng.permutation(33)
    yield "path in random order", 33, perm[path(33)]
    yield "ring 64", 64, np.concatenate([path(64), [[63, 0]]])
    yield "two rings and a lone node", 31, np.concatenate([path(12), [[11, 0]], 12 + path(18), [[29, 12]]])
    yield "star", 12, np.stack([np.zeros(11, int), np.arange(1, 12)], 1)
    yield "complete 7", 7, np.array([(i, j) for i in range(7) for j in range(i)])
    yield ("grid 9x13",) + _grid(9, 13)
    yield "random tree", 40, np.array([(rng.integers(0, k), k) for k in range(1, 40)])
    yield "random sparse", 50, rng.integers(0, 50, (70, 2))
    yield "double edges", 6, np.concatenate([path(6), path(6)])


@pytest.mark.parametrize("name,n,edges", list(_graphs()), ids=[g[0] for g in _graphs()])
def test_plan_solves_like_the_whole_system(host, name, n, edges):
    e = np.ascontiguousarray([x for x in np.asarray(edges).reshape(-1, 2) if x[0] != x[1]], np.int32).reshape(-1, 2)
    out = np.zeros(3, np.int32)
    for max_w, max_dense in ((148, 2048), (148, 0), (2, 0), (2, 36)):
        r = host.host_cond_residual(n, len(e), e.ctypes.data_as(ctypes.c_void_p), max_w, max_dense, 5,
                                    out.ctypes.data_as(ctypes.c_void_p))
        assert r <= 1e-12, f"{name}: {r}"
        assert 0 <= out[0] < n


def test_stent_condenses_onto_its_crossings(host, scenes):
    """A braided stent keeps at most its crossings; a wire keeps one or two nodes."""
    conf, _, _ = scenes.braided_stent(wires=16, elems_per_wire=60, crossing_every=5)
    e = np.ascontiguousarray(conf.beams.conn, np.int32)
    out = np.zeros(3, np.int32)
    r = host.host_cond_residual(len(conf.nodes), len(e), e.ctypes.data_as(ctypes.c_void_p), 148, 0, 5,
                                out.ctypes.data_as(ctypes.c_void_p))
    crossings = int((np.bincount(e.ravel()) == 4).sum())
    assert r <= 1e-12 and len(conf.nodes) - out[0] <= crossings
