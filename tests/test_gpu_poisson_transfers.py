"""The standalone solve's host arrays: moved in place by the SMs from 65,536 cells on, by copies below and where the
arrays are not aligned to whole doubles. Either way the result is the same, and the source is left as it was. (Two solves
are not the same bits: the mean that the result leaves with is summed in the order in which blocks finish, so it may differ
by eps |p| for each of the blocks.)"""
import ctypes as C

import numpy as np
import pytest

from atsat_gb300 import abi, dyn, synth
from helpers import case

pytestmark = pytest.mark.gpu


def at_offset(a, nbytes):
    """A copy of `a` that starts nbytes past an allocation's own alignment."""
    buf = np.zeros(a.nbytes + 64, dtype=np.uint8)
    start = (-buf.ctypes.data) % 16 + nbytes
    view = np.frombuffer(buf.data, dtype=np.float64, count=a.size, offset=start)
    view[:] = a.reshape(-1)
    return buf, buf.ctypes.data + start


# 65,148, 65,880 and 66,612 cells, odd and even row lengths; sources and results on and off 16-byte boundaries, and unaligned
@pytest.mark.parametrize("offsets", [(0, 0), (8, 0), (0, 8), (8, 8), (4, 4)], ids=str)
@pytest.mark.parametrize("shape", [(12, 61, 89), (12, 61, 90), (12, 61, 91)], ids=str)
def test_in_place_and_copied(shape, offsets):
    g, P, _ = case(shape, seed=3)
    double = C.POINTER(C.c_double)
    out = []
    with dyn.Dycore(g, P) as d:
        src = d.poisson_project(synth.poisson_source(g, seed=5))
        for direct in (False, True):
            d.set_host_direct(direct)
            hold, s = at_offset(src, offsets[0])
            room, p = at_offset(np.full(g.shape, np.nan), offsets[1])
            before = hold.copy()
            st = abi.PoissonStats()
            rc = dyn.lib().atsat_dyn_poisson_solve(d.h, 3, C.cast(s, double), C.cast(p, double), 0.0, 1, 0, 1.0, C.byref(st))
            assert rc == abi.OK
            assert np.array_equal(hold, before)
            out.append(np.frombuffer(room.data, dtype=np.float64, count=src.size, offset=p - room.ctypes.data).copy())
    blocks = -(-g.km // 32) * -(-g.jm // 8) * -(-(g.im - 2) // 8)
    bar = blocks * np.finfo(float).eps * np.max(np.abs(out[0]))
    assert np.isfinite(out[0]).all() and np.max(np.abs(out[0] - out[1])) <= bar
