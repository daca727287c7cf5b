"""What the tuner's cache holds for one x solve is not taken for another: the y solves of the transposed frame need
an x solve that hands the fields over, which k_solve_xs does not."""
import numpy as np
import pytest

import oracle
from nemaktis_gb300 import _lib, api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 1e-4)])
@pytest.mark.parametrize("first,then", [(None, "xs:M=32:KS=1;auto"), ("xw:M=8:KS=2:W=3;auto", "xs:M=32:KS=1;auto"),
                                        ("xs:M=32:KS=1;auto", "xw:M=8:KS=1:W=3;auto"), ("auto;yx:M=4:KS=2", None),
                                        (None, "auto;yx:M=4:KS=2")])
def test_a_cached_direction_fits_the_other_one(gpu, first, then, precision, tol):
    js, lc, shape = case((600, 120, 4), q=((0.0, 0.0), (0.03, 0.01)), seed=5, smooth=True, NA=0.4137)
    ref = np.zeros(shape, np.complex128)
    oracle.run_backend_without_mask(js, lc, ref)
    _lib.load().nbpm_tune_cache_clear()
    for cfg in (first, then):
        out = np.zeros(shape, np.complex128)
        with api.Plan([{"json": js, "lc": lc, "E": out}], precision=precision, solve_config=cfg) as p:
            x, y = p.solve_config(0)[0].split(";")
            assert not (y.startswith("yx") and x.startswith("xs"))
            p.upload()
            p.execute()
            p.download()
        assert rel_l2(out, ref) <= tol
