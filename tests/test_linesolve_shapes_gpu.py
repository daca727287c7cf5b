"""Periodic line solves over the shapes that take another route: fewer unknowns than a chunk, ragged and full
last chunks, one to eight warps a line, lines past shared memory, and systems that are not diagonally
dominant, whose chunks are not joined. Tolerance 1e-12 as for the other line-solve tests."""
import numpy as np
import pytest

from nemaktis_gb300 import _lib  # noqa: F401  (the gpu fixture loads the library)
from tests.test_linesolve_gpu import dense_reference, gpu_solve, periodic_systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nlines", [(4, 1), (5, 7), (6, 2), (9, 3), (33, 5), (128, 4), (129, 700), (130, 3),
                                      (513, 3), (514, 9), (1025, 2), (1500, 2)])
def test_shapes(gpu, L, nlines):
    s = periodic_systems(L, nlines, seed=L + nlines)
    x, ref = gpu_solve(gpu.nbpm_periodic_tridiag_solve, *s), dense_reference(*s)
    assert np.linalg.norm(x - ref) / np.linalg.norm(ref) < 1e-12


@pytest.mark.parametrize("L", [2049, 2100, 3600])
def test_long_lines(gpu, L):
    """Against the residual of the systems: ||A x - b|| <= 1e-12 ||b||."""
    inf, mid, sup, rhs = periodic_systems(L, 2, seed=L)
    x = gpu_solve(gpu.nbpm_periodic_tridiag_solve, inf, mid, sup, rhs)
    n = L - 1
    y, b = x[:, :n], rhs[:, :n]
    r = inf[:, :n] * np.roll(y, 1, 1) + mid[:, :n] * y + sup[:, :n] * np.roll(y, -1, 1) - b
    assert np.linalg.norm(r) / np.linalg.norm(b) < 1e-12
    assert np.array_equal(x[:, n], x[:, 0])


@pytest.mark.parametrize("L", [9, 65, 257])
def test_weak_diagonal(gpu, L):
    """Lines whose couplings exceed the diagonal (strong skew coupling, well conditioned) beside dominant ones."""
    inf, mid, sup, rhs = periodic_systems(L, 6, seed=L)
    inf[::2] = -3.0 + 0.1 * inf[::2]
    sup[::2] = 3.0 + 0.1 * sup[::2]
    x, ref = gpu_solve(gpu.nbpm_periodic_tridiag_solve, inf, mid, sup, rhs), dense_reference(inf, mid, sup, rhs)
    assert np.linalg.norm(x - ref) / np.linalg.norm(ref) < 1e-12
