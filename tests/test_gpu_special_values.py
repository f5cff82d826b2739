"""States with values that the integer comparisons of the FP64 kernels have to sort as the reference's comparisons do:
NaN, infinities, negative zero, temperatures at and below zero and beyond the reciprocal's FP32 range, negative k* and
omega*, sources at and beyond their clips. Planted in single cells, so that their stencils' neighbours see them too; every
field has to agree with the oracle in its finite cells to the FP64 bar and be the same elsewhere. (Infinities stand where the
reference bounds or tests them. In an advected field their differences cancel to NaN or not by the order of the sums.)"""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import TOL_FP64, case
from oracle import oracle

pytestmark = pytest.mark.gpu

NAN, INF = np.nan, np.inf
PLANTS = {
    "nue": {F.NUE: [NAN, INF, -INF, -0.0, -1.0e-3, 5.0e-324]},
    "temperature": {F.T: [-0.0, 0.0, -1.0, 1.0e-40, 1.0e40, 1.0e-300]},
    "temperature_nan": {F.T: [NAN]},
    "turbulence": {F.TKE: [-0.0, -1.0e-3, 1.0e-30, 0.0], F.DIS: [-0.0, -1.0, 1.0e-12, 1.0e30]},
    "heat": {F.Q_PRECIP: [1.0e9, -1.0e9, NAN, INF], F.Q_RAD: [1.0e9, -1.0e9, -INF, NAN]},
    "density": {F.RHO_MIX: [0.0, -1.0, NAN, INF, 1.0e-320]},
    "cloud": {F.H2O_CLOUD: [-0.0, NAN, -1.0e-3], F.CH4_ICE: [-1.0, 1.0e-9, NAN]},
    "winds": {F.U: [30.0, NAN], F.W: [-0.0, -30.0]},
}


def planted(name, shape, **over):
    g, P, st = case(shape, seed=6, **over)
    n = 0
    for f, values in PLANTS[name].items():
        for v in values:
            st.arrays[f][2 + n % (g.im - 4), 3 + (2 * n) % (g.jm - 6), (5 * n) % (g.km - 1)] = v
            n += 1
        if f < F.NPROG:
            st.arrays[F.N_BASE + f] = st.arrays[f].copy()
    return g, P, st


def agree(got, ref, fields, what):
    bad = []
    with np.errstate(invalid="ignore", over="ignore"):
        for f in fields:
            a, b = got[f], ref[f]
            finite = np.isfinite(b)
            same = np.array_equal(a[~finite], b[~finite], equal_nan=True)
            err = np.max(np.abs(a[finite] - b[finite]), initial=0.0)
            if not (same and err <= TOL_FP64 * np.max(np.abs(b[finite]), initial=0.0)):
                bad.append((F.NAMES[f], bool(same), err))
    assert not bad, (what, bad)


@pytest.mark.parametrize("over", [{}, {"rad_coupling": 1.0}, {"buoy_legacy": 1, "turb_coupling": 0.5}],
                         ids=lambda o: ",".join(o) or "default")
@pytest.mark.parametrize("name", sorted(PLANTS))
def test_right_hand_side(name, over):
    g, P, st = planted(name, (9, 13, 35), **over)
    ref = st.copy()
    oracle.rhs(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.set_write_all_rhs(True)
        d.computeBuoyancyRefLevel()
        d.computeMetricPressure()
        d.RHSSat_pass()
        d.download(list(range(F.NFIELDS)))
    agree(got.arrays, ref.arrays, F.RHS_FIELDS + [F.AUX_U, F.AUX_V, F.AUX_W], f"{name} {over}")


@pytest.mark.parametrize("name", sorted(PLANTS))
def test_level_mean(name):
    g, P, st = planted(name, (9, 13, 35))
    want = oracle.buoyancy_ref_level(st.copy(), P)
    with dyn.Dycore(g, P) as d:
        d.load_state(st)
        d.computeBuoyancyRefLevel()
        got = d.buoy_ref_level()
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    f = np.isfinite(want)
    assert np.max(np.abs(got[f] - want[f])) <= TOL_FP64 * np.max(np.abs(want[f]))


@pytest.mark.parametrize("over", [{}, {"turb_free": 0}, {"buoy": 2}], ids=lambda o: ",".join(o) or "default")
@pytest.mark.parametrize("name", sorted(PLANTS))
def test_closure(name, over):
    from atsat_gb300 import abi
    g, P, st = planted(name, (9, 13, 35))
    tp = abi.make_turb_params(**over)
    ref = st.copy()
    oracle.turbulence(ref, P, tp)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.set_turb_params(tp)
        d.TurbulenceSat_run()
        d.download(list(range(F.NFIELDS)))
    agree(got.arrays, ref.arrays, [F.TKE, F.DIS, F.NUE, F.TKE_SOURCE, F.DIS_SOURCE], f"{name} {over}")


@pytest.mark.parametrize("knobs", [{}, {"press_line": 1}, {"press_incr": 0}, {"press_src": 0, "press_incr": 0}],
                         ids=lambda o: ",".join(o) or "default")
@pytest.mark.parametrize("value", [NAN, INF, -INF, -0.0, 1.0e300, 5.0e-324], ids=repr)
def test_pressure(value, knobs):
    g, P, st = case((9, 13, 35), seed=6, **knobs)
    for f in (F.RHS_V, F.AUX_V):
        st.arrays[f][4, 6, 7] = value
    ref = st.copy()
    want = oracle.pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        stats = d.PressureSolver_run()
        d.download([F.P_DYN])
    agree(got.arrays, ref.arrays, [F.P_DYN], f"{value} {knobs}")
    assert stats.src_clamped == want.src_clamped
