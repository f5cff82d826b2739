"""The FP64 stage kernel's instances against the oracle: default switches and couplings (branches compiled out), each
switch and coupling that selects the general instance, unequal Schmidt numbers, and the tendencies written or not, at
grids around its 32 x 4 blocks."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import TOL_FP64, case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu

KNOBS = [{}, {"sc_nh3": 0.7}, {"precip_coupling": 0.5}, {"chemical_reaction": 2.0}, {"turb_coupling": 0.25},
         {"species_divu": 1.0}, {"rad_coupling": 1.0}, {"thermal_massflux": 1.0}, {"buoy_legacy": 1},
         {"metric_split": 0, "coriolis_split": 0}, {"turb_active": 0}]


@pytest.mark.parametrize("knobs", KNOBS, ids=lambda k: "-".join(k) or "default")
@pytest.mark.parametrize("shape", [(5, 9, 33), (7, 12, 34), (6, 13, 66)], ids=str)
def test_step_matches_the_oracle(shape, knobs):
    g, P, st = case(shape, seed=5, **knobs)
    ref = st.copy()
    oracle.rk4_step(ref, P)
    out = {}
    for every in (False, True):
        got = st.copy()
        with dyn.Dycore(g, P) as d:
            d.load_state(got)
            d.set_write_all_rhs(every)
            d.RungeKuttaSat()
            d.download(list(range(F.NFIELDS)))
        compare(got.arrays, ref.arrays, F.PROG + [F.RHS_U, F.RHS_V, F.RHS_W, F.AUX_U, F.AUX_V, F.AUX_W]
                + (F.RHS_FIELDS if every else []), TOL_FP64, f"{shape} {knobs} all rhs {every}")
        out[every] = got.arrays
    # the tracers' weighted and centred sums differ by the rounding of weight times value: with dt sum|weight| < 1
    # on these grids (Courant number), a few units in the last place of the field's largest value over four stages
    eps = np.finfo(np.float64).eps
    for q in F.PROG:
        a, b = out[False][q], out[True][q]
        assert np.max(np.abs(a - b)) <= 16 * eps * np.max(np.abs(b)), F.NAMES[q]
