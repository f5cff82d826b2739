"""Grids whose tracer tiles run as two field groups, and the grids on either side of that line (114 and 228 tiles): the
march variant against the oracle (one step, the mixed path's 1e-6 bar), its tracers against the direct kernel (1e-7)."""
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu


def step(g, P, st, variant):
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.set_stage_variant(variant)
        d.RungeKuttaSat()
        d.download(list(range(F.NFIELDS)))
    return got.arrays


# tiles: 108 (four groups), 120, 135, 196 (two), 240 (one)
@pytest.mark.parametrize("over", [{}, {"turb_active": 0}], ids=["turb", "no_turb"])
@pytest.mark.parametrize("shape", [(26, 49, 97), (40, 25, 100), (61, 40, 60), (30, 36, 224), (31, 121, 61)], ids=str)
def test_two_groups(shape, over):
    g, P, st = case(shape, seed=4, precision=1, **over)
    ref = st.copy()
    oracle.rk4_step(ref, P)
    march = step(g, P, st, dyn.Dycore.STAGE_MARCH)
    compare(march, ref.arrays, F.PROG, 1e-6, f"march {shape}")
    compare(march, step(g, P, st, dyn.Dycore.STAGE_DIRECT), F.PROG[F.H2O:], 1e-7, f"march against direct {shape}")
