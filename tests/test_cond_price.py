"""The condensation plan never costs more, by its own prices, than the band of the whole system: also where the
elimination does not come down to a system that can be inverted (nets of more than 41 a side), whose levels make
the band wider, its LU dearer and its blocks too large to stage."""
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MAX_W, MAX_DENSE, STAGE_B = 148, 2048, 594


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    so = str(tmp_path_factory.mktemp("plan") / "plan_host.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", os.path.join(HERE, "host", "plan_host.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)

    def f(a, b):
        out, cost = (ctypes.c_int * 3)(), (ctypes.c_double * 2)()
        lib.host_grid_plan(a, b, MAX_W, MAX_DENSE, STAGE_B, out, cost)
        return list(out), list(cost)

    return f


@pytest.mark.parametrize("a,b", [(42, 42), (43, 43), (44, 44), (48, 48), (50, 50), (60, 60), (64, 64), (100, 100),
                                 (20, 200), (30, 200), (40, 60), (16, 500), (40, 500)])
def test_condensed_band_costs_no_more_than_the_whole_band(plan, a, b):
    (kept, bw, _), (mine, whole) = plan(a, b)
    assert kept > MAX_DENSE and bw <= 6 * MAX_W + 5
    assert mine <= whole


@pytest.mark.parametrize("a,b,levels,kept", [(12, 12, 1, 492), (20, 20, 2, 960), (33, 33, 6, 1578), (41, 41, 10, 1962), (10, 400, 25, 1500)])
def test_plans_that_reach_the_inverse(plan, a, b, levels, kept):
    """These systems are inverted; their plans (and so their results' bits) do not hang on the band's price.  12 x 12: a
    level, without which 1,024 of them invert five times as much."""
    out, _ = plan(a, b)
    assert (out[0], out[2]) == (kept, levels)
