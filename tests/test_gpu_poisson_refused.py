"""A direct solve on a ring beyond the transforms' shared memory (4693 meridians in FP64, 9386 in FP32) is refused with a
status. Nothing that reads the caller's source may be left on the stream when the call returns: the source's memory is
unmapped right after it, and the handle goes on to other solves."""
import ctypes as C
import mmap

import numpy as np
import pytest

from atsat_gb300 import abi, dyn, synth
from helpers import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,km", [(3, 4801), (4, 9601), (5, 9601)], ids=["direct64", "direct32", "refine_direct"])
def test_refused_solve_leaves_the_source_alone(method, km):
    g, P, _ = case((5, 7, km), seed=3)
    src = synth.poisson_source(g, seed=5)
    double = C.POINTER(C.c_double)
    with dyn.Dycore(g, P) as d:
        for _ in range(3):
            room = mmap.mmap(-1, src.nbytes)
            view = np.frombuffer(room, dtype=np.float64)
            view[:] = src.reshape(-1)
            p = np.zeros(g.shape)
            st = abi.PoissonStats()
            rc = dyn.lib().atsat_dyn_poisson_solve(d.h, method, C.cast(view.ctypes.data, double), abi.dptr(p), 1e-10, 5, 0, 1.0,
                                                   C.byref(st))
            assert rc == abi.E_CUDA
            del view
            room.close()
        q, st = d.poisson_solve("sor64", src, tol=0.0, max_iter=2)
    assert np.isfinite(q).all() and st["iterations"] == 2
