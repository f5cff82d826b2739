"""The tracer kernel's tiles (64 x 4 x 4 or 32 x 8 x 4 cells, whichever pads less) and stream at the sizes where they can go wrong: rings around one and two
tiles' width (the periodic partner inside the box, in the seam box, alone in a tile), rows and levels that leave a
remainder, the fields with two sources at couplings other than 1, without turbulence, in the march and tiled2 variants.
One step, its tracers against the direct kernel (1e-7: the same FP32 arithmetic, differently contracted) and all
prognostic fields against the oracle (the mixed path's 1e-6 bar)."""
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


@pytest.mark.parametrize("over", [{}, {"turb_active": 0}, {"precip_coupling": 0.7, "chemical_reaction": 1.3}],
                         ids=["default", "no_turb", "couplings"])
@pytest.mark.parametrize("shape", [(5, 9, 17), (6, 8, 64), (7, 10, 65), (8, 11, 66), (9, 12, 68), (10, 13, 69),
                                   (11, 14, 70), (6, 9, 129), (7, 11, 134),
                                   (5, 8, 33), (6, 11, 36), (7, 12, 128), (8, 10, 126), (5, 11, 193)], ids=str)
def test_tiles_match_direct_and_oracle(shape, over):
    g, P, st = case(shape, seed=8, precision=1, **over)
    ref = st.copy()
    oracle.rk4_step(ref, P)
    direct = step(g, P, st, dyn.Dycore.STAGE_DIRECT)
    for name in ("MARCH", "TILED2"):
        got = step(g, P, st, getattr(dyn.Dycore, "STAGE_" + name))
        compare(got, direct, F.PROG[F.H2O:], 1e-7, f"{name} against direct {shape}")
        compare(got, ref.arrays, F.PROG, 1e-6, f"{name} {shape}")
