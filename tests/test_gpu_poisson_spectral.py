"""The spectral direct solve at ring lengths of every radix (2, 3, 4, 5, larger primes, a prime ring), odd and even
radial row counts, against the sparse CPU solve; radial systems between and beyond the register layouts' steps.

Bars: the operator's conditioning bounds an FP64 solve (test_gpu_poisson.py: 1e-8 on the solution, 1e-10 on the
residual); the refinement stops at 1e-10 or stalls at the FP64 solve's own residual."""
import numpy as np
import pytest

import poisson_ref as PR
from helpers import case

pytestmark = pytest.mark.gpu

# rings 8, 9, 12, 14, 25, 30, 37, 49, 60, 64, 77; radial rows 3 .. 12
SHAPES = [(5, 9, 9), (6, 8, 10), (7, 11, 13), (8, 10, 15), (9, 12, 26), (10, 9, 31), (11, 13, 38), (12, 11, 50),
          (13, 14, 61), (14, 9, 65), (9, 10, 78)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_direct_and_refine(shape):
    from atsat_gb300 import dyn, synth
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
    n = g.km - 1
    assert abs(p[1:-1, 1:-1, :n].mean()) <= 1e-12 * scale and abs(q[1:-1, 1:-1, :n].mean()) <= 1e-12 * scale


# radial rows at the layouts' steps (10, 20, 40 FP64; 24, 40, 80 FP32) and beyond. The bar is the a-priori bound of the
# elimination's backward error: each of its 2 NJ steps adds the rounding of sums of NI + 2 terms relative to |L| |p|
@pytest.mark.parametrize("im", [12, 13, 22, 23, 26, 27, 42, 43, 82, 84])
def test_radial_layouts(im):
    from atsat_gb300 import dyn, synth
    shape = (im, 7, 9)
    g, P, _ = case(shape, seed=3)
    A, _ = PR.matrix(g, P)
    with dyn.Dycore(g, P) as d:
        src = d.poisson_project(synth.poisson_source(g, seed=5))
        p, _ = d.poisson_solve("direct64", src)
        p32, s32 = d.poisson_solve("direct32", src)
    rows, f = (im - 2) + 2, PR.to_vec(g, src)
    bound = 2 * 5 * rows * np.linalg.norm(abs(A) @ np.abs(PR.to_vec(g, p))) / np.linalg.norm(f)
    assert PR.rel_residual(g, A, p, src) <= bound * np.finfo(np.float64).eps
    assert s32["rel_residual"] <= max(1.0, bound * np.finfo(np.float32).eps)
    assert np.isfinite(p32).all()
