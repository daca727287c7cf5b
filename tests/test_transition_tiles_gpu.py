"""The transition's tiles of 32 x 32 points, clipped to the plane: planes that end one point before, on and after a
tile and after a segment of 8 columns or 4 rows, with one axis too short to be filtered, and shifts of either sign.
FP64 against the oracle with the bound of the parity tests (1e-10); FP32 on pairs and on single slots against FP64
within 1e-5 (rounding 6e-8 times some hundred operations in sequence per slab)."""
import numpy as np
import pytest

import oracle
from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(31, 33), (32, 32), (33, 31), (64, 65), (65, 34), (40, 37), (41, 36), (97, 75), (3, 45), (45, 2), (4, 4)])
def test_clipped_tiles(gpu, dims):
    js, lc, shape = case((*dims, 4), q=((0.3, -0.2), (-0.25, 0.35)), seed=sum(dims), smooth=True)
    ref, e64, e32, e32s = (np.zeros(shape, np.complex128) for _ in range(4))
    oracle.run_backend_without_mask(js, lc, ref)
    api.run(js, lc, e64, precision="fp64")
    assert rel_l2(e64, ref) <= 1e-10
    api.run(js, lc, e32, precision="fp32")
    assert rel_l2(e32, e64) <= 1e-5
    if min(dims) > 3:
        M = [next(m for m in (2, 3, 4) if 32 * m >= n - 1) for n in dims]
        api.run(js, lc, e32s, precision="fp32", solve_config="xc:M=%d:KS=1;yx:M=%d:KS=1" % tuple(M))
        assert rel_l2(e32s, e64) <= 1e-5
        api.run(js, lc, e32s, precision="fp32", solve_config="xc:M=%d:KS=2;yx:M=%d:KS=2" % tuple(M))
        assert rel_l2(e32s, e64) <= 1e-5
