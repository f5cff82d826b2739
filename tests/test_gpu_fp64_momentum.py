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


@pytest.mark.parametrize("over", [{}, {"metric_split": 0, "coriolis_split": 0}, {"species_divu": 1.0}],
                         ids=lambda o: ",".join(o) or "default")
def test_aux_does_not_see_the_pressure_gradient(over):
    """aux_u, aux_v, aux_w are the tendencies without the gradient of p_dyn. Formed as the tendency plus that gradient,
    they carry its rounding, which is large against them where the gradient is; so they are the same bits at any p_dyn."""
    g, P, st = case((7, 12, 34), seed=4, **over)
    a = rhs_pass(g, P, st)
    strong = st.copy()
    strong.arrays[F.P_DYN] *= 1.0e3
    b = rhs_pass(g, P, strong)
    for aux, rhs in ((F.AUX_U, F.RHS_U), (F.AUX_V, F.RHS_V), (F.AUX_W, F.RHS_W)):
        assert np.array_equal(a[aux], b[aux]), F.NAMES[aux]
        assert not np.array_equal(a[rhs], b[rhs])
