"""The partitioned line solves (chunks factored by themselves, joined through their border unknowns) where
they can go wrong: lines that end on, just before and just after a chunk or warp, the shortest lines, and
couplings from weak to so strong that the joining iterates for long or the line is solved as one chunk.

FP64 against the oracle with the bound of the parity tests (1e-10): the joining is exact to rounding (2^-57
of the border unknowns) and the line operators, 1 + i*(positive semi-definite), do not amplify."""
import numpy as np
import pytest

import oracle
from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10
Q2 = ((0.0, 0.0), (0.1, -0.05))


def run_both(dims, cfg, **kw):
    js, lc, shape = case(dims, q=Q2, seed=sum(dims), **kw)
    ref, out = np.zeros(shape, np.complex128), np.zeros(shape, np.complex128)
    oracle.run_backend_without_mask(js, lc, ref)
    api.run(js, lc, out, precision="fp64", solve_config=cfg)
    return rel_l2(out, ref)


# n = N - 1 unknowns per line: 3, 4 (two chunks), one chunk more or less than a warp, ragged last chunks
@pytest.mark.parametrize("n,M", [(3, 2), (4, 2), (63, 2), (64, 2), (65, 4), (127, 4), (129, 8), (249, 8), (256, 8),
                                 # odd chunks (no padding in shared memory), and twice the shortest (half the lanes idle)
                                 (74, 3), (96, 3), (129, 5), (160, 5), (161, 6), (192, 6), (193, 7), (224, 7), (63, 4), (96, 6)])
def test_chunk_edges_one_warp(gpu, n, M):
    cfg = "xc:M=%d:KS=%d;yx:M=%d:KS=%d"
    assert run_both((n + 1, 6, 4), cfg % (M, 2, 2, 2)) <= FP64_TOL
    assert run_both((6, n + 1, 4), cfg % (2, 1, M, 1)) <= FP64_TOL


# several warps per line: the last chunk at a warp's first lane, mid-warp, at a warp's last lane
@pytest.mark.parametrize("n,W", [(257, 2), (265, 2), (512, 2), (513, 3), (1000, 4)])
def test_chunk_edges_several_warps(gpu, n, W):
    assert run_both((n + 1, 5, 3), "xw:M=8:KS=2:W=%d;yx:M=2:KS=1" % W) <= FP64_TOL
    assert run_both((5, n + 1, 3), "xc:M=2:KS=1;yx:M=8:KS=1:W=%d" % W) <= FP64_TOL


# transverse spacings from a quarter wavelength down to where a line is one chunk (coupling ~ dz / dx^2)
@pytest.mark.parametrize("dx", [0.25, 0.05, 0.02, 0.004])
@pytest.mark.parametrize("dims,cfg", [((70, 12, 4), "xc:M=4:KS=2;yx:M=2:KS=2"), ((12, 300, 3), "xc:M=2:KS=1;yx:M=8:KS=2:W=2"),
                                      ((300, 12, 3), "xw:M=8:KS=1:W=2;yx:M=2:KS=1")])
def test_strong_coupling(gpu, dims, cfg, dx):
    assert run_both(dims, cfg, spacings=(dx, dx, 0.25), smooth=True) <= FP64_TOL
