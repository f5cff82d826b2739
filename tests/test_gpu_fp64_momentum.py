"""Properties of the FP64 momentum tendencies that rounding must not cost."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import case

pytestmark = pytest.mark.gpu


def rhs_pass(g, P, st):
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.computeBuoyancyRefLevel()
        d.computeMetricPressure()
        d.RHSSat_pass()
        d.download(list(range(F.NFIELDS)))
    return got.arrays


@pytest.mark.parametrize("shape", [(5, 9, 33), (7, 12, 34), (11, 40, 67)], ids=str)
def test_no_zonal_coriolis_force_on_the_held_means(shape):
    """u and v at the means that the phi Coriolis term holds, uniform along phi, and w = 0: every term of rhs_w is zero,
    the Coriolis term as a difference of equal values."""
    g, P, st = case(shape, seed=4, turb_active=0)
    rng = np.random.default_rng(2)
    for f, table in ((F.U, st.cell_ubar0), (F.V, st.cell_vbar0)):
        table[...] = rng.normal(0.0, 0.1, table.shape)
        st.arrays[f][...] = table[:, :, None]
    for f in (F.W, F.P_DYN):
        st.arrays[f][...] = 0.0
    a = rhs_pass(g, P, st)
    assert np.all(a[F.RHS_W][1:-1, 2:-2, :-1] == 0.0)
    assert np.any(a[F.RHS_V][1:-1, 2:-2, :-1] != 0.0)
