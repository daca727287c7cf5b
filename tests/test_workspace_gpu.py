"""Solves do not depend on what the device memory of their workspace held before: memory full of NaN is given back just
before the plan allocates. Configurations are forced, so that no timing run writes the workspace first; lines that leave
threads past their last chunk, joined by Jacobi steps and by scans."""
import ctypes

import numpy as np
import pytest

import oracle
from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu


def runtime():
    try:
        return ctypes.CDLL("libcudart.so")
    except OSError:
        return ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")


@pytest.fixture
def dirty_memory(gpu):
    """Buffers of many sizes, set to bytes of 0xff (NaN in either precision); every other one is given back, so that
    the blocks they are cut from stay and what is cut from them next holds those bytes."""
    rt = runtime()
    held = []
    for k in range(2000):
        p = ctypes.c_void_p()
        size = 8192 << (k // 2 % 8)  # 8 KB .. 1 MB, in pairs
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        assert rt.cudaMemset(p, 0xFF, ctypes.c_size_t(size)) == 0
        held.append(p)
    assert rt.cudaDeviceSynchronize() == 0
    for p in held[::2]:
        assert rt.cudaFree(p) == 0
    yield
    for p in held[1::2]:
        rt.cudaFree(p)


@pytest.mark.parametrize("dx", [0.25, 0.03])
@pytest.mark.parametrize("n,m,cfg", [(33, 8, "xc:M=2:KS=2;yx:M=2:KS=2"), (20, 9, "xc:M=2:KS=1;yx:M=2:KS=1"), (97, 50, "xc:M=8:KS=1;yx:M=4:KS=1"), (120, 66, "xc:M=8:KS=2;yx:M=4:KS=2"),
                                     (270, 12, "xw:M=8:KS=2:W=2;yx:M=2:KS=2"), (530, 9, "xw:M=8:KS=1:W=3;yx:M=2:KS=1")])
def test_what_the_memory_held_does_not_matter(dirty_memory, n, m, cfg, dx):
    js, lc, shape = case((n + 1, m + 1, 3), q=((0.0, 0.0), (0.1, -0.05)), seed=n, smooth=True, spacings=(dx, dx, 0.25), NA=0.4137)
    ref = np.zeros(shape, np.complex128)
    oracle.run_backend_without_mask(js, lc, ref)
    for precision, tol in (("fp64", 1e-10), ("fp32", 1e-4)):
        out = np.zeros(shape, np.complex128)
        api.run(js, lc, out, precision=precision, solve_config=cfg)
        assert rel_l2(out, ref) <= tol
