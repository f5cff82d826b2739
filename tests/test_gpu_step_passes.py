"""The once-a-step passes where their code depends on the size or the switches: the radial boundary conditions by form
(shells below eight levels take the steps in order), the level mean's rows and the metric scan's levels around their
batches, and the mixed path's frozen terms with the switches off their defaults. Against the oracle."""
import numpy as np
import pytest

from atsat_gb300 import dyn, fields as F
from helpers import case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu

ALL = list(range(F.NFIELDS))


# products and sums of two or three terms, and one quotient: a few ulps against the oracle
@pytest.mark.parametrize("shape", [(5, 7, 9), (7, 8, 130), (8, 9, 17), (9, 13, 131)], ids=str)
@pytest.mark.parametrize("over", [dict(), dict(bc_radius_form=1, bc_bottom_form=2), dict(bc_radius_form=3, bc_bottom_form=1),
                                  dict(bc_radius_form=0, bc_bottom_form=0, bc_lid_u=0, bc_top_taper=0),
                                  dict(bc_radius_form=2, bc_bottom_form=3, bc_lid_u=0, bc_top_taper=1),
                                  dict(bc_species_lid_copy=0, bc_species_wall_copy=0),
                                  dict(bc_species_lid_copy=0, bc_species_wall_copy=1),
                                  dict(bc_species_lid_copy=1, bc_species_wall_copy=0, turb_active=0),
                                  dict(bc_species_wall_copy=2, local_rho=0)],
                         ids=lambda d: ",".join(f"{k}={v}" for k, v in d.items()) or "default")
def test_radial_boundary(shape, over):
    g, P, st = case(shape, seed=31, **over)
    ref = st.copy()
    oracle.boundary_conditions(ref, P)
    s = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(s)
        d.boundary_conditions()
        d.download(ALL)
    compare(s.arrays, ref.arrays, ALL, 1e-13, f"bc {shape} {over}")


# rows per chunk 0..23, radial levels around the batches of eight; sums of positive terms in another order than the
# oracle's
@pytest.mark.parametrize("shape", [(5, 7, 9), (9, 40, 33), (10, 160, 130), (17, 273, 20), (18, 360, 16)], ids=str)
def test_level_mean_and_metric_scan(shape):
    g, P, st = case(shape, seed=32)
    ref = st.copy()
    oracle.steps(ref, P, 1)
    s = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(s)
        d.iterate(1, 1)
        d.download(ALL)
    compare(s.arrays, ref.arrays, [F.P_METRIC, F.RHS_U, F.RHS_V, F.U], 1e-12, f"step {shape}")


# one mixed step, the mixed path's 1e-6 bar
@pytest.mark.parametrize("over", [dict(), dict(coriolis_split=0), dict(metric_split=0, coriolis_split=0),
                                  dict(buoy_legacy=1)],
                         ids=lambda d: ",".join(f"{k}={v}" for k, v in d.items()) or "default")
def test_mixed_frozen_terms(over):
    g, P, st = case((9, 31, 61), seed=33, precision=1, **over)
    ref = st.copy()
    oracle.rk4_step(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.RungeKuttaSat()
        d.download(ALL)
    compare(got.arrays, ref.arrays, F.PROG, 1e-6, f"mixed {over}")
    assert all(np.isfinite(got.arrays[q]).all() for q in F.PROG)
