"""Caps outside the sensible range: the clamps compare bit patterns, which order like the numbers only where both are
non-negative. A cap of zero, negative zero, a negative one, NaN and infinity act as the reference's comparisons do."""
import math

import numpy as np
import pytest

from atsat_gb300 import abi, dyn, fields as F
from helpers import TOL_FP64, case
from oracle import oracle

pytestmark = pytest.mark.gpu


def agree(got, ref, what):
    """The FP64 bar on the finite values; the others the same."""
    finite = np.isfinite(ref)
    assert np.array_equal(got[~finite], ref[~finite], equal_nan=True), what
    size = np.max(np.abs(ref), where=finite, initial=0.0)
    assert np.max(np.abs(got[finite] - ref[finite]), initial=0.0) <= TOL_FP64 * size, what


@pytest.mark.parametrize("over", [{}, {"press_src": 0, "press_incr": 0}, {"press_incr": 0}], ids=lambda o: ",".join(o) or "default")
@pytest.mark.parametrize("cap", [0.0, -0.0, -1.0e-9, -0.2, math.nan, -math.nan, math.inf, -math.inf], ids=repr)
def test_source_cap(cap, over):
    g, P, st = case((9, 13, 17), seed=9, pdyn_cap=cap, **over)
    ref = st.copy()
    want = oracle.pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        stats = d.PressureSolver_run()
        d.download([F.P_DYN])
    agree(got.arrays[F.P_DYN], ref.arrays[F.P_DYN], f"cap {cap} {over}")
    assert stats.src_clamped == want.src_clamped


@pytest.mark.parametrize("over", [{}, {"turb_free": 0}, {"abl_taper": 1}], ids=lambda o: ",".join(o) or "default")
@pytest.mark.parametrize("cap", [0.0, -0.0, 1.0e-3, -1.0, math.nan, -math.nan, math.inf, -math.inf], ids=repr)
def test_viscosity_cap(cap, over):
    g, P, st = case((6, 8, 34), seed=35)
    tp = abi.make_turb_params(nue_max_phys=cap, **over)
    ref = st.copy()
    prod, _ = oracle.turbulence(ref, P, tp)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.set_turb_params(tp)
        d.TurbulenceSat_run()
        d.download(list(range(F.NFIELDS)))
        p, _ = d.turbulence_diag()
    for f in (F.TKE, F.DIS, F.NUE, F.TKE_SOURCE, F.DIS_SOURCE):
        agree(got.arrays[f], ref.arrays[f], f"{F.NAMES[f]} {cap} {over}")
    agree(p, prod, f"P_k {cap} {over}")
