"""atsat_dyn_set_write_all_rhs asks for more output; it must not change the run. The state after a step and after
iterations is the same bits with it on and off, for the FP64 stage kernel's instances and the mixed variants."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import case

pytestmark = pytest.mark.gpu

STATE = F.PROG + [F.P_DYN, F.RHS_U, F.RHS_V, F.RHS_W, F.AUX_U, F.AUX_V, F.AUX_W]


@pytest.mark.parametrize("over", [{}, {"sc_nh3": 0.7}, {"precip_coupling": 0.5, "chemical_reaction": 2.0}, {"species_divu": 1.0},
                                  {"rad_coupling": 1.0, "thermal_massflux": 1.0}, {"turb_active": 0},
                                  {"metric_split": 0, "coriolis_split": 0}, {"precision": 1}],
                         ids=lambda o: ",".join(o) or "default")
@pytest.mark.parametrize("shape", [(7, 12, 34), (27, 40, 66)], ids=str)
def test_the_state_is_the_same(shape, over):
    g, P, st = case(shape, seed=5, **over)
    out = []
    for every in (False, True):
        got = st.copy()
        with dyn.Dycore(g, P) as d:
            d.load_state(got)
            d.set_write_all_rhs(every)
            d.RungeKuttaSat()
            d.restoreVar()
            d.iterate(0, 2)
            d.download(STATE)
        out.append(got.arrays)
    changed = [F.NAMES[f] for f in STATE if not np.array_equal(out[0][f], out[1][f], equal_nan=True)]
    assert not changed, changed
