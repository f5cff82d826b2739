"""The march variant on grids around its launch rules: the tracers' field groups (13, 4 and 1 blocks per tile) and the
fused stage launch, against the oracle (one step, the mixed path's 1e-6 bar on every prognostic field); the tracers, whose launch the rules change, also
against the direct kernel (1e-7)."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu


def step(g, P, st, variant, iterations):
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.set_stage_variant(variant)
        if iterations:
            d.iterate(0, iterations)
        else:
            d.RungeKuttaSat()
        d.download(list(range(F.NFIELDS)))
    return got.arrays


# tiles of 32 x 8 x 4 cells: 1 (13 groups), 54, 70, 216 (4 groups), 252 (one); odd rings among them
@pytest.mark.parametrize("over", [{}, {"turb_active": 0}], ids=["turb", "no_turb"])
@pytest.mark.parametrize("shape", [(5, 9, 17), (22, 13, 225), (26, 28, 66), (18, 52, 289), (26, 53, 193)], ids=str)
def test_groups_match_oracle_and_direct(shape, over):
    g, P, st = case(shape, seed=4, precision=1, **over)
    ref = st.copy()
    oracle.rk4_step(ref, P)
    march = step(g, P, st, dyn.Dycore.STAGE_MARCH, 0)
    compare(march, ref.arrays, F.PROG, 1e-6, f"march {shape}")
    direct = step(g, P, st, dyn.Dycore.STAGE_DIRECT, 0)
    compare(march, direct, F.PROG[F.H2O:], 1e-7, f"march against direct {shape}")


@pytest.mark.parametrize("shape", [(9, 31, 61), (21, 60, 121)], ids=str)
def test_resident_iterations_with_groups(shape):
    g, P, st = case(shape, seed=6, precision=1)
    ref = st.copy()
    oracle.steps(ref, P, 4, iter0=0)
    got = step(g, P, st, dyn.Dycore.STAGE_MARCH, 4)
    compare(got, ref.arrays, F.PROG + [F.P_DYN], 1e-6, f"march {shape}")
    assert all(np.isfinite(got[q]).all() for q in F.PROG)
