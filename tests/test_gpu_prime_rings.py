"""Rings whose largest prime factor exceeds what a warp's lanes take in one round (64): the transforms run a block per row
pair. Around that line, with other radices beside the prime, few and many rows. The bars are those of the spectral solve's
and the pressure pass's own tests."""
import numpy as np
import pytest

import poisson_ref as PR
from atsat_gb300 import dyn, fields as F, synth
from helpers import TOL_FP64, case, compare
from oracle import oracle

pytestmark = pytest.mark.gpu

# rings 61, 67, 134, 179, 201, 284
SHAPES = [(6, 9, 62), (5, 9, 68), (6, 8, 135), (7, 11, 180), (8, 9, 202), (5, 10, 285)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_direct_and_refine(shape):
    g, P, _ = case(shape, seed=3)
    A, _ = PR.matrix(g, P)
    with dyn.Dycore(g, P) as d:
        src = d.poisson_project(synth.poisson_source(g, seed=5))
        x = PR.solve(g, A, src)
        p, st = d.poisson_solve("direct64", src)
        q, sr = d.poisson_solve("refine_direct", src, tol=1e-10, max_iter=30)
    scale = np.max(np.abs(x))
    assert np.max(np.abs(PR.to_vec(g, p) - x)) <= 1e-8 * scale
    assert PR.rel_residual(g, A, p, src) <= 1e-9
    assert sr["rel_residual"] <= max(1e-10, 10 * st["rel_residual"])
    assert np.max(np.abs(PR.to_vec(g, q) - x)) <= 1e-8 * scale


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_barotropic(shape):
    g, P, st = case(shape, seed=8, press_baro=1)
    ref = st.copy()
    oracle.pressure(ref, P)
    got = st.copy()
    with dyn.Dycore(g, P) as d:
        d.load_state(got)
        d.PressureSolver_run()
        d.download([F.P_DYN])
    compare(got.arrays, ref.arrays, [F.P_DYN], TOL_FP64, str(shape))
