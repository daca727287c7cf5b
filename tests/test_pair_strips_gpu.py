"""Right-hand sides formed in strips of 4 and 2 lines: plane heights from the smallest
on, with every remainder of a strip, and strips that hold the periodic line and its copy in every place. FP32 mode
against FP64, bound 1e-5: rounding 6e-8 times some hundred operations in sequence per slab."""
import numpy as np
import pytest

from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [4, 5, 6, 7, 8, 9, 12, 13])
@pytest.mark.parametrize("n,cfg", [(60, "xc:M=2:KS=2"), (181, "xc:M=6:KS=2"), (256, "xc:M=8:KS=2"), (401, "xw:M=8:KS=2:W=2")])
def test_strip_heights(gpu, n, ny, cfg):
    js, lc, shape = case((n + 1, ny, 4), q=((0.1, -0.05),), seed=n + ny, smooth=True)
    e64, e32 = np.zeros(shape, np.complex128), np.zeros(shape, np.complex128)
    api.run(js, lc, e64, precision="fp64")
    api.run(js, lc, e32, precision="fp32", solve_config=cfg + ";yx:M=2:KS=2")
    assert rel_l2(e32, e64) <= 1e-5
    # the y direction takes the same lines from the transposed frame
    js, lc, shape = case((ny, n + 1, 4), q=((0.1, -0.05),), seed=n + ny, smooth=True)
    e64, e32t = np.zeros(shape, np.complex128), np.zeros(shape, np.complex128)
    api.run(js, lc, e64, precision="fp64")
    api.run(js, lc, e32t, precision="fp32", solve_config="xc:M=2:KS=2;" + cfg.replace("xc", "yx").replace("xw", "yx"))
    assert rel_l2(e32t, e64) <= 1e-5
