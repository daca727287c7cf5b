"""Lines whose chunks are coupled strongly (transverse spacings far below a wavelength, a last chunk of one point) take
about the time of weakly coupled ones: they are joined by scans, whatever the coupling. Also the edges of that
join: lines of one, two and three chunks, chunks that end on a warp, and several warps."""
import time

import numpy as np
import pytest

import oracle
from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu

Q2 = ((0.0, 0.0), (0.1, -0.05))


def execute_ms(dims, precision, spacing, cfg=None):
    js, lc, shape = case(dims, q=Q2, seed=1, smooth=True, spacings=(spacing, spacing, 0.25))
    with api.Plan([{"json": js, "lc": lc, "E": np.zeros(shape, np.complex128)}], precision=precision, solve_config=cfg) as p:
        p.upload()
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            p.execute()
            t.append(time.perf_counter() - t0)
    return 1e3 * min(t)


# by the time of a line joined in a few steps; one thread per line took 3 to 6 times as long
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", [(64, 64, 16), (129, 129, 12), (256, 256, 8), (512, 512, 8)])
def test_time_does_not_depend_on_the_coupling(gpu, dims, precision):
    weak = execute_ms(dims, precision, 0.25)
    for spacing in (0.05, 0.02):
        assert execute_ms(dims, precision, spacing) <= 2.0 * weak, spacing


# n unknowns in chunks of M: one chunk, two, three; last chunk of one point; the last lane; W warps
@pytest.mark.parametrize("n,cfg", [(4, "xc:M=4:KS=1"), (6, "xc:M=4:KS=2"), (9, "xc:M=4:KS=1"), (97, "xc:M=4:KS=2"), (63, "xc:M=2:KS=2"),
                                   (64, "xc:M=2:KS=1"), (255, "xc:M=8:KS=1"), (257, "xw:M=8:KS=1:W=2"), (505, "xw:M=8:KS=2:W=2"),
                                   (512, "xw:M=8:KS=2:W=2"), (513, "xw:M=8:KS=1:W=3"), (1023, "xw:M=8:KS=1:W=4")])
@pytest.mark.parametrize("dx", [0.25, 0.03, 0.005])
def test_join_edges(gpu, n, cfg, dx):
    kw = dict(q=Q2, seed=n, smooth=True, spacings=(dx, dx, 0.25))
    js, lc, shape = case((n + 1, 6, 3), **kw)
    ref, out, out32 = (np.zeros(shape, np.complex128) for _ in range(3))
    oracle.run_backend_without_mask(js, lc, ref)
    api.run(js, lc, out, precision="fp64", solve_config=cfg + ";yx:M=2:KS=1")
    assert rel_l2(out, ref) <= 1e-10  # as for the parity tests
    api.run(js, lc, out32, precision="fp32", solve_config=cfg.replace("KS=1", "KS=2") + ";yx:M=2:KS=2")
    assert rel_l2(out32, ref) <= 1e-4  # the FP32 mode's bound
    js, lc, shape = case((6, n + 1, 3), **kw)
    ref, out = np.zeros(shape, np.complex128), np.zeros(shape, np.complex128)
    oracle.run_backend_without_mask(js, lc, ref)
    api.run(js, lc, out, precision="fp64", solve_config="xc:M=2:KS=2;yx" + cfg[2:])
    assert rel_l2(out, ref) <= 1e-10
