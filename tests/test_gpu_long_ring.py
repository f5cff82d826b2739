"""PRESS_BAROTROPIC around the longest ring that the transforms hold in shared memory (4693 meridians): the transforms up
to it, sums over the meridians beyond. Against the oracle at the FP64 bar."""
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import TOL_FP64, case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("km", [4681, 4694, 4695, 4702])
def test_long_ring(km):
    g, P, st = case((5, 7, km), seed=8, press_baro=1)
    ref = st.copy()
    oracle.pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.PressureSolver_run()
        d.download([F.P_DYN])
    compare(got.arrays, ref.arrays, [F.P_DYN], TOL_FP64, f"ring of {km - 1}")
