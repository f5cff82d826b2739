"""The mode solve's wide kernel (radial rows beyond the register layouts): its batches around their lengths, blocks of up to
and of more than 256 rows, in both precisions. The bar is the a-priori bound of the elimination's backward error: each of
its 2 NJ steps adds the rounding of sums of NI + 2 terms relative to |L| |p|."""
import numpy as np
import pytest

import poisson_ref as PR
from atsat_gb300 import dyn, synth
from helpers import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im", [59, 82, 83, 130, 258, 259, 300])
def test_wide_blocks(im):
    g, P, _ = case((im, 7, 9), seed=3)
    A, _ = PR.matrix(g, P)
    with dyn.Dycore(g, P) as d:
        src = d.poisson_project(synth.poisson_source(g, seed=5))
        p, _ = d.poisson_solve("direct64", src)
        q, _ = d.poisson_solve("direct32", src)
    for x, eps in ((p, np.finfo(np.float64).eps), (q, np.finfo(np.float32).eps)):
        bound = 2 * 5 * im * np.linalg.norm(abs(A) @ np.abs(PR.to_vec(g, x))) / np.linalg.norm(PR.to_vec(g, src))
        assert PR.rel_residual(g, A, x, src) <= bound * eps
