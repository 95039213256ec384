"""Node state as it is read back (gathered by a kernel in chunks of 4096 nodes) against what was
assigned: a simulation smaller than a chunk, one of more than one chunk, second of a batch, some
fields only.  Copies, so bits are equal."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FIELDS = ("u", "ud", "udd", "w", "wd", "wdd", "R", "dR")


@pytest.mark.parametrize("wires,epw", [(16, 8), (32, 171)])
def test_state_round_trip(eb, scenes, wires, epw):
    built = [scenes.braided_stent(wires=16, elems_per_wire=11, grid=None),
             scenes.braided_stent(wires=wires, elems_per_wire=epw, grid=None)]
    eng = eb.GpuSimulations([b[0] for b in built], built[0][1], [b[2] for b in built])
    n = len(built[1][0].nodes)
    assert (n > 4096) == (wires == 32)
    rng = np.random.default_rng(n)
    new = {k: rng.standard_normal((n, 9 if k in ("R", "dR") else 3)) for k in FIELDS}
    first = eng.state(0)
    eng.set_state(1, **new)
    for at_n in (False, True):
        got = eng.state(1, at_n=at_n)
        assert all(np.array_equal(got[k], new[k]) for k in FIELDS)
    assert all(np.array_equal(eng.state(0)[k], first[k]) for k in FIELDS)
    # two fields only
    ud, dR = np.zeros((n, 3)), np.zeros((n, 9))
    P = C.POINTER(C.c_double)
    rc = eng.L.eb_get_state(eng.h, 1, None, ud.ctypes.data_as(P), None, None, None, None, None, dR.ctypes.data_as(P))
    assert rc == 0 and np.array_equal(ud, new["ud"]) and np.array_equal(dR, new["dR"])
    eng.close()
