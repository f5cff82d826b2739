"""PRESS_BAROTROPIC with rows of very unequal strength: a source in one row of latitude alone, in one zonal mode, so that
the correction falls off by many orders over theta. The reference drops the modes below 1e-12 of a row's own sum, which
keeps the other modes exactly zero in every row; noise of a strong row in its weak neighbours' modes would not be dropped
and, in a low mode, outlast the correction itself. So each row is held to the FP64 bar relative to its own largest value
(the elimination's recurrences have terms of one sign: a few units in the last place a row)."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import TOL_FP64, case
from oracle import oracle

pytestmark = pytest.mark.gpu


# rings with a radix whose twiddled sums of equal values round (7, 5, 11), a partner row on either side of the strong
# one, an even and an odd number of rows
@pytest.mark.parametrize("row", [7, 8])
@pytest.mark.parametrize("shape", [(7, 62, 29), (7, 62, 61), (6, 63, 45)], ids=str)
def test_weak_rows_beside_a_strong_one(shape, row):
    g, P, st = case(shape, seed=1, press_baro=1)
    for f in range(F.NFIELDS):
        st.arrays[f] = np.zeros(g.shape)
    ring = np.arange(g.km) % (g.km - 1)
    st.arrays[F.RHS_W][:, row, :] = 1e-3 * np.array([0.0, 1.0, 0.0, -1.0])[ring % 4]
    ref = st.copy()
    oracle.pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.PressureSolver_run()
        d.download([F.P_DYN])
    p, q = got.arrays[F.P_DYN], ref.arrays[F.P_DYN]
    size = np.max(np.abs(q), axis=(0, 2))
    assert size.max() > 1e3 * size[-1] > 0.0
    err = np.max(np.abs(p - q), axis=(0, 2))
    assert np.all(err <= TOL_FP64 * size), (err / size).max()
