"""The metric pressure scan takes the levels above the first in batches of four: every remainder, with and without p_baro,
against the oracle (a trapezoid sum in the same order, products contracted differently)."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("baro", [False, True], ids=["plain", "p_baro"])
@pytest.mark.parametrize("im", [5, 6, 7, 8, 9, 10, 11, 12])
def test_remainders(im, baro):
    g, P, st = case((im, 8, 35), seed=32)
    if baro:
        st.p_baro = np.random.default_rng(im).normal(0.0, 1.0e-3, g.shape)
    ref = st.copy()
    oracle.metric_pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.computeMetricPressure()
        d.download([F.P_METRIC])
    assert np.any(ref.arrays[F.P_METRIC] != 0.0)
    compare(got.arrays, ref.arrays, [F.P_METRIC], 1e-14, f"{im} {baro}")
