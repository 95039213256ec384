"""Launch rules that need no GPU (csrc/eb_launch_rules.hpp)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    so = str(tmp_path_factory.mktemp("rules") / "rules_host.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", os.path.join(HERE, "host", "rules_host.cpp"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def test_solver_cta_is_whole_warps(rules):
    """A warp owns whole chunks of the vectors: with no whole warp the solver's loops would not advance,
    with a partial one two warps would own the same chunk."""
    f = rules.host_gmres_cta_threads
    assert [f(t) for t in (-7, 0)] == [0, 0]
    for t in range(1, 513):
        assert f(t) % 32 == 0 and max(64, t) <= f(t) <= max(64, t + 31)
    assert f(513) < 0 and f(1024) < 0


def test_state_is_read_on_the_handles_device(rules):
    """eb_get_state launches: the handle's device is current during the call, the caller's afterwards."""
    out = (ctypes.c_int * 2)()
    for caller, device, sets in ((0, 0, 0), (1, 0, 2), (0, 3, 2)):
        assert rules.host_on_device(caller, device, out) == device
        assert list(out) == [caller, sets]
    csrc = os.path.join(HERE, "..", "endobeams.jl_gb300", "csrc", "eb_abi.cu")
    body = open(csrc).read().split("static int get_state_impl(", 1)[1].split("launch_state(", 1)[0]
    assert "OnDevice<CudaDevice> on(h->device)" in body


def test_element_launches_follow_the_devices_size(rules):
    """Thirty elements a CTA beyond twenty per SM; the two passes side by side unless both have thirty elements a
    CTA and fewer than two CTAs per SM."""
    wide = lambda n, sms: bool(rules.host_wide_elements(ctypes.c_int64(n), sms))
    beside = lambda b, c, n, sms: bool(rules.host_side_by_side(b, c, ctypes.c_int64(n), sms))
    for sms in (152, 148, 76):
        assert [bool(rules.host_many_elements(ctypes.c_int64(n), sms)) for n in (448 * sms, 448 * sms + 1)] == [False, True]
        assert [wide(n, sms) for n in (0, 20 * sms, 20 * sms + 1)] == [False, False, True]
        assert [beside(3, 3, n, sms) for n in (60 * sms - 1, 60 * sms)] == [False, True]
        assert beside(3, 1, 60 * sms - 1, sms) and beside(1, 3, 60 * sms - 1, sms) and beside(1, 1, 1, sms)


def test_preconditioners_that_do_not_fit(rules):
    """Inverses give way to the bands of the same kept nodes, the largest saving first; only where the bands do
    not fit either does everything become block-Jacobi."""
    jacobi, band, inverse = 0, 1, 2

    def fit(sims, kinds, room):
        n = len(sims)
        b = (ctypes.c_int64 * (3 * n))(*[x for s in sims for x in s])
        k = (ctypes.c_int32 * n)(*kinds)
        rules.host_fit_precond(n, b, ctypes.c_int64(room), k)
        return list(k)

    sims = [(10, 20, 100), (10, 30, 200), (10, 0, 50), (10, 90, 80), (5, 40, 0), (1000, 1000, 1000)]
    want = [inverse, inverse, inverse, inverse, band, jacobi]
    full = 4 * 10 + 100 + 200 + 50 + 80 + 45
    assert fit(sims, want, full) == want
    assert fit(sims, want, full - 1) == [inverse, band, inverse, inverse, band, jacobi]
    assert fit(sims, want, full - 170) == [inverse, band, inverse, inverse, band, jacobi]
    assert fit(sims, want, full - 171) == [band, band, inverse, inverse, band, jacobi]
    assert fit(sims, want, full - 250) == [band, band, inverse, inverse, band, jacobi]
    assert fit(sims, want, full - 251) == [jacobi] * 6


@pytest.mark.parametrize("n,b", [(64, 11), (192, 5), (198, 11), (320, 64), (320, 65), (334, 129), (600, 200), (600, 599)])
def test_inversion_leaves_out_zero_blocks_only(rules, n, b):
    """Blocked in-place Gauss-Jordan (64-wide pivots) of a band matrix: with the blocks past dense_reach left
    out every value is that of the full steps."""
    rng = np.random.default_rng(n + b)
    i, j = np.indices((n, n))
    ld = -(-n // 64) * 64
    full = np.eye(ld)
    full[:n, :n] = np.where(abs(i - j) <= b, rng.standard_normal((n, n)), 0.0) + 3.0 * np.sqrt(2 * b + 1) * np.eye(n)
    cut, nb = full.copy(), ld // 64
    blk = lambda M, r, c: M[64 * r:64 * r + 64, 64 * c:64 * c + 64]
    want = np.linalg.inv(full)
    for M, reach in ((full, lambda k: nb), (cut, lambda k: min(nb, rules.host_dense_reach(k, b)))):
        for k in range(nb):
            D, m = np.linalg.inv(blk(M, k, k)), reach(k)
            assert m > k + 1 or k + 1 == nb  # the next pivot block is updated
            C = {r: blk(M, r, k) @ D for r in range(m) if r != k}
            O = {c: blk(M, k, c).copy() for c in range(m) if c != k}
            for r in range(m):
                for c in range(m):
                    if r == k:
                        blk(M, r, c)[:] = D if c == k else D @ O[c]
                    elif c == k:
                        blk(M, r, c)[:] = -C[r]
                    else:
                        blk(M, r, c)[:] -= C[r] @ O[c]
    assert np.array_equal(full, cut)
    assert np.abs(cut - want).max() <= 1e-12 * np.abs(want).max() * n


@pytest.mark.parametrize("sims", [[(1, 5)], [(15, 125), (30, 479)], [(30, 479), (0, 593), (3, 11), (9, 1000)], [(0, 0)], [(32, 2041)]])
def test_grids_of_the_inversion_hold_every_simulations_blocks(rules, sims):
    """sims: blocks a side (0: not inverted) and half bandwidth.  Every block that a step changes has a CTA, the next
    pivot block among them, and a step has no more rows of CTAs than its widest simulation."""
    n, side = len(sims), (ctypes.c_int * 64)()
    got = rules.host_dense_grids(n, (ctypes.c_int * n)(*[a for a, _ in sims]), (ctypes.c_int * n)(*[b for _, b in sims]), side)
    assert got == max(a for a, _ in sims)
    for k in range(got):
        rows = [min(a, rules.host_dense_reach(k, b)) for a, b in sims if k < a]
        assert side[k] == max(rows) and all(r > k + 1 or k + 1 == a for r, (a, _) in zip(rows, [x for x in sims if k < x[0]]))


@pytest.mark.parametrize("sms", [1, 76, 152])
def test_inversions_of_many_tiles(rules, sms):
    assert [bool(rules.host_dense_many(ctypes.c_int64(n), sms)) for n in (1, 80 * sms, 80 * sms + 1)] == [False, False, True]
