"""The FP32 solves and transitions on pairs of slots, forced, against the FP64 result: lines that end on, before
and after a chunk or a warp, plane heights that leave a block of lines part-filled, one and several pairs
and wavelengths, normal incidence alone (no shift) and tilted, and couplings strong enough for many joining steps and
for single-chunk lines. Bound 1e-4, the FP32 mode's; the few slabs of these cases keep FP32 within 1e-5 (rounding
6e-8 times some hundred operations in sequence per slab)."""
import numpy as np
import pytest

from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu

Q0 = ((0.0, 0.0),)
Q3 = ((0.0, 0.0), (0.1, -0.05), (-0.2, 0.15))


def check(dims, cfg, q=Q3, tol=1e-5, **kw):
    js, lc, shape = case(dims, q=q, seed=sum(dims), smooth=True, **kw)
    e64, e32 = np.zeros(shape, np.complex128), np.zeros(shape, np.complex128)
    api.run(js, lc, e64, precision="fp64")
    api.run(js, lc, e32, precision="fp32", solve_config=cfg)
    assert rel_l2(e32, e64) <= tol


@pytest.mark.parametrize("n,m,M", [(3, 4, 2), (63, 9, 2), (64, 64, 2), (65, 6, 4), (128, 7, 4), (129, 10, 8), (256, 5, 8),
                                   (74, 5, 3), (96, 6, 3), (129, 7, 5), (191, 4, 6), (224, 5, 7),
                                   (257, 6, 16), (500, 4, 16)])
@pytest.mark.parametrize("q", [Q0, Q3])
def test_one_warp_per_line(gpu, n, m, M, q):
    other = 2
    check((n + 1, m + 1, 4), "xc:M=%d:KS=2;yx:M=%d:KS=2" % (M, other), q)
    check((m + 1, n + 1, 4), "xc:M=%d:KS=2;yx:M=%d:KS=2" % (other, M), q)


@pytest.mark.parametrize("n,m,W", [(257, 4, 2), (265, 7, 2), (512, 5, 2), (513, 4, 3), (1023, 6, 4), (1800, 4, 8)])
@pytest.mark.parametrize("q", [Q0, Q3])
def test_several_warps_per_line(gpu, n, m, W, q):
    check((n + 1, m + 1, 3), "xw:M=8:KS=2:W=%d;yx:M=2:KS=2" % W, q)
    check((m + 1, n + 1, 3), "xc:M=2:KS=2;yx:M=8:KS=2:W=%d" % W, q)


def test_several_wavelengths_and_passes(gpu):
    js, lc, shape = case((40, 37, 6), wavelengths=(0.45, 0.55, 0.65), q=Q3, seed=5, smooth=True)
    e64, e32, e32p = (np.zeros(shape, np.complex128) for _ in range(3))
    cfg = "xc:M=2:KS=2;yx:M=2:KS=2"
    api.run(js, lc, e64, precision="fp64")
    api.run(js, lc, e32, precision="fp32", solve_config=cfg)
    api.run(js, lc, e32p, precision="fp32", solve_config=cfg, groups_per_pass=2)
    assert rel_l2(e32, e64) <= 1e-5
    np.testing.assert_array_equal(e32, e32p)


@pytest.mark.parametrize("dx", [0.05, 0.02, 0.004])
@pytest.mark.parametrize("dims,cfg", [((70, 12, 4), "xc:M=4:KS=2;yx:M=2:KS=2"),
                                      ((300, 12, 3), "xw:M=8:KS=2:W=2;yx:M=2:KS=2")])
def test_strong_coupling(gpu, dims, cfg, dx):
    check(dims, cfg, spacings=(dx, dx, 0.25), tol=1e-4)
