"""PRESS_LINE and PRESS_BAROTROPIC at ring lengths of every radix of the transforms (2, 3, 4, 5, larger primes, a prime
ring), odd and even row counts, and the smallest radial systems, against the oracle at the FP64 bar."""
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import TOL_FP64, case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knobs", [{"press_baro": 1}, {"press_line": 1, "press_baro": 1, "press_sweeps": 2}, {"press_line": 1}],
                         ids=["baro", "both", "line"])
@pytest.mark.parametrize("shape", [(5, 7, 9), (5, 8, 10), (6, 9, 13), (7, 10, 26), (8, 11, 38), (9, 12, 50), (10, 13, 61),
                                   (11, 14, 129), (6, 37, 78)], ids=str)
def test_pressure_call(shape, knobs):
    g, P, st = case(shape, seed=8, **knobs)
    ref = st.copy()
    oracle.pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.PressureSolver_run()
        d.download([F.P_DYN])
    compare(got.arrays, ref.arrays, [F.P_DYN], TOL_FP64, f"{shape} {knobs}")
