"""Periodic line solves whose right-hand sides span many orders of magnitude, hold a NaN, or whose last chunk is short:
every unknown is exact relative to itself, and the time does not depend on the remainder."""
import ctypes
import time

import numpy as np
import pytest

from nemaktis_gb300 import _lib
from tests.test_linesolve_gpu import gpu_solve

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def systems(L, nlines, seed, c=0.15):
    """1 + i * (second difference with weights near c)."""
    rng = np.random.default_rng(seed)
    a, b = (c * (1 + 0.2 * rng.uniform(-1, 1, (nlines, L))) for _ in range(2))
    return -1j * a, 1 + 1j * (a + b), -1j * b


def reference(inf, mid, sup, rhs):
    """Solution in extended precision: the line opened at its first unknown, x_0 = 1 and the right-hand side as two
    solves of the other unknowns by sweeps."""
    inf, mid, sup, b = (np.asarray(v[:, :-1], np.clongdouble).copy() for v in (inf, mid, sup, rhs))
    n = b.shape[1]
    unit = np.zeros_like(b)
    unit[:, 1] -= inf[:, 1]
    unit[:, n - 1] -= sup[:, n - 1]
    cols = np.stack([b, unit])
    beta, d = mid.copy(), cols.copy()
    for i in range(2, n):
        l = inf[:, i] / beta[:, i - 1]
        beta[:, i] = mid[:, i] - l * sup[:, i - 1]
        d[:, :, i] -= l * d[:, :, i - 1]
    y = np.zeros_like(cols)
    y[:, :, n - 1] = d[:, :, n - 1] / beta[:, n - 1]
    for i in range(n - 2, 0, -1):
        y[:, :, i] = (d[:, :, i] - sup[:, i] * y[:, :, i + 1]) / beta[:, i]
    p, u = y
    x0 = (b[:, 0] - inf[:, 0] * p[:, -1] - sup[:, 0] * p[:, 1]) / (mid[:, 0] + inf[:, 0] * u[:, -1] + sup[:, 0] * u[:, 1])
    x = p + x0[:, None] * u
    x[:, 0] = x0
    return np.concatenate([x, x[:, :1]], 1)


@pytest.mark.parametrize("L", [66, 130, 250, 513, 1025])
def test_right_hand_sides_of_one_point(gpu, L):
    """A right-hand side of one point decays along the line by about 7 per point; allowed is 32 eps per point passed."""
    inf, mid, sup = systems(L, 5, L)
    rhs = np.zeros((5, L), complex)
    for k, i in enumerate((1, 7, (L - 1) // 2, L - 3, L - 2)):
        rhs[k, i] = 1 + 0.5j
    x, ref = gpu_solve(gpu.nbpm_periodic_tridiag_solve, inf, mid, sup, rhs), reference(inf, mid, sup, rhs)
    big = np.abs(ref) > 1e-290
    assert (np.abs(x - ref)[big] <= 32 * EPS * L * np.abs(ref)[big]).all()


@pytest.mark.parametrize("L", [66, 250, 513])
def test_a_large_value_among_small_ones(gpu, L):
    rng = np.random.default_rng(L)
    inf, mid, sup = systems(L, 4, L)
    rhs = 1 + rng.uniform(0, 1, (4, L)) + 0j
    rhs[np.arange(4), [0, 5, L // 2, L - 2]] = 1e20
    x, ref = gpu_solve(gpu.nbpm_periodic_tridiag_solve, inf, mid, sup, rhs), reference(inf, mid, sup, rhs)
    # a value's own terms, and what reaches it of its neighbours'
    size = np.abs(ref) + 0.15 * (np.abs(np.roll(ref[:, :-1], 1, 1)) + np.abs(np.roll(ref[:, :-1], -1, 1)))[:, list(range(L - 1)) + [0]]
    assert (np.abs(x - ref) <= 32 * EPS * L * size).all()


@pytest.mark.parametrize("L", [66, 257, 513, 1025])
def test_nan_reaches_its_whole_line(gpu, L):
    inf, mid, sup = systems(L, 3, L)
    rhs = np.ones((3, L), complex)
    rhs[1, L // 3] = np.nan
    x = gpu_solve(gpu.nbpm_periodic_tridiag_solve, inf, mid, sup, rhs)
    assert np.isnan(x[1]).all() and np.isfinite(x[[0, 2]]).all()


@pytest.mark.parametrize("n", [2500, 2501, 2560, 2561, 2750, 2751])
def test_longest_lines(gpu, n):
    inf, mid, sup = systems(n + 1, 2, n)
    rng = np.random.default_rng(n)
    rhs = rng.normal(size=(2, n + 1)) + 0j
    x, ref = gpu_solve(gpu.nbpm_periodic_tridiag_solve, inf, mid, sup, rhs), reference(inf, mid, sup, rhs)
    assert np.linalg.norm(x - ref) <= 1e-14 * np.linalg.norm(ref)


def solve_us(lib, L, nlines):
    torch = pytest.importorskip("torch")
    inf, mid, sup = systems(L, nlines, 1)
    dev = [torch.from_numpy(v).cuda() for v in (inf, mid, sup, np.ones((nlines, L), complex))]
    x = torch.zeros_like(dev[3])
    t = []
    for _ in range(6):
        t0 = time.perf_counter()
        _lib.check(lib.nbpm_periodic_tridiag_solve(L, nlines, *[ctypes.c_void_p(v.data_ptr()) for v in dev],
                                                   ctypes.c_void_p(x.data_ptr()), None))
        t.append(time.perf_counter() - t0)
    return 1e6 * min(t)


# last chunks of one point and full ones; by one thread per line the former took 7 to 30 times as long
@pytest.mark.parametrize("ragged,full,nlines", [(250, 257, 2000), (50, 49, 4096), (98, 97, 1000), (66, 65, 650), (514, 513, 2048)])
def test_time_does_not_depend_on_the_remainder(gpu, ragged, full, nlines):
    assert solve_us(gpu, ragged, nlines) <= 3.0 * solve_us(gpu, full, nlines)
