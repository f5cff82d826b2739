"""The SST source kernel's branches against the oracle: blending settled by the bounds (the default, y* of 1e20 m) and
evaluated (wall distances), the taper's separate passes, every buoyancy mode, at grids around its 32 x 4 blocks. The bars
are those of the closure's own tests."""
import pytest

from test_gpu_fp64 import _turbulence_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [{}, {"turb_free": 0}, {"abl_taper": 1}, {"buoy": 2}, {"buoy": 1, "turb_free": 0}, {"curv": 0}],
                         ids=lambda o: ",".join(f"{k}={v}" for k, v in o.items()) or "default")
@pytest.mark.parametrize("shape", [(5, 7, 9), (6, 8, 34), (7, 13, 66)], ids=str)
def test_sst_branches(shape, over):
    _turbulence_case(shape, over)
