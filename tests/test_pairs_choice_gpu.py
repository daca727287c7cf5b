"""Which FP32 configurations run on pairs of slots: x and y solves with two slots per thread and chunks of at most 8
points, unless the x part says ":single". The two families sum the Woodbury iterates in another order, so that their
results differ in the last bits, which tells them apart."""
import numpy as np
import pytest

from nemaktis_gb300 import _lib, api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu

Q3 = ((0.0, 0.0), (0.1, -0.05), (-0.2, 0.15))


def run(dims, cfg, precision="fp32"):
    js, lc, shape = case(dims, q=Q3, seed=sum(dims), smooth=True)
    E = np.zeros(shape, np.complex128)
    api.run(js, lc, E, precision=precision, solve_config=cfg)
    return E


@pytest.mark.parametrize("dims,x,y", [((40, 37, 4), "xc:M=2:KS=2", "yx:M=2:KS=2"), ((64, 64, 4), "xc:M=2:KS=2", "yx:M=2:KS=2"),
                                      ((97, 75, 4), "xc:M=3:KS=2", "yx:M=3:KS=2"), ((258, 30, 4), "xw:M=8:KS=2:W=2", "yx:M=2:KS=2"),
                                      ((30, 600, 4), "xc:M=2:KS=2", "yx:M=8:KS=2:W=3"), ((256, 256, 4), "xc:M=8:KS=2", "yx:M=8:KS=2")])
def test_single_forces_the_general_kernels(gpu, dims, x, y):
    e64 = run(dims, None, "fp64")
    pairs, single = run(dims, x + ";" + y), run(dims, x + ":single;" + y)
    assert not np.array_equal(pairs, single)
    assert rel_l2(pairs, e64) <= 1e-5 and rel_l2(single, e64) <= 1e-5
    # the mark means nothing where there are no pairs
    assert np.array_equal(run(dims, x + ":single;" + y, "fp64"), run(dims, x + ";" + y, "fp64"))


@pytest.mark.parametrize("dims", [(40, 24, 5), (64, 64, 5), (200, 150, 4)])
@pytest.mark.parametrize("half", [None, "xc:M=%d:KS=2;auto", "auto;yx:M=%d:KS=2"])
def test_the_tuners_choice_is_what_runs(gpu, dims, half):
    n = dims[0 if half and half[0] == "x" else 1] - 1
    cfg0 = half and half % next(m for m in (2, 3, 4, 5, 6, 7, 8) if 32 * m >= n)
    js, lc, shape = case(dims, q=Q3, seed=3, smooth=True)
    _lib.load().nbpm_tune_cache_clear()
    seen = []
    for _ in range(2):
        E = np.zeros(shape, np.complex128)
        with api.Plan([{"json": js, "lc": lc, "E": E}], precision="fp32", solve_config=cfg0) as p:
            cfg, report = p.solve_config(0)
            p.upload()
            p.execute()
            p.download()
        seen.append((cfg, E))
        x, y = cfg.split(";")
        could = ":KS=2" in x and not x.startswith("xs") and y.startswith("yx") and y.endswith(":KS=2")
        if "pairs slower" in report:
            assert not could or x.endswith(":single")
        elif "pairs " in report:
            assert could and not x.endswith(":single") and "pairs " + cfg in report
    assert seen[0][0] == seen[1][0] and "cached" in report
    forced = np.zeros(shape, np.complex128)
    api.run(js, lc, forced, precision="fp32", solve_config=seen[0][0])
    assert np.array_equal(forced, seen[0][1]) and np.array_equal(forced, seen[1][1])
