"""Fourier transforms with large prime factors and the column-wise screen filter: mesh sizes that are
prime, twice or three times a prime, and whose column groups are ragged, with apertures that keep few, some and most
columns; the screen filter against the oracle, the focus against numpy. Bounds: those of the parity tests
(FP64 1e-10, FP32 1e-4), and 1e-12 for the focus as for the other microscope tests."""
import numpy as np
import pytest

import oracle
from nemaktis_gb300 import api
from oracle import micrograph
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(97, 11, 3), (13, 101, 3), (22, 33, 3), (121, 34, 2), (5, 4, 3), (130, 17, 2), (10, 194, 2)])
@pytest.mark.parametrize("NA", [0.05, 0.45, 0.98])
def test_screen_filter(gpu, dims, NA):
    kw = dict(q=((0.0, 0.0), (0.12, -0.07)), NA=NA, iso_thick=(1.0,), iso_index=(1.4,), z_shift=0.3, nout="1.1")
    js, lc, shape = case(dims, seed=7, smooth=True, **kw)
    ref, out, out32 = (np.zeros(shape, np.complex128) for _ in range(3))
    oracle.run_backend_without_mask(js, lc, ref)
    api.run(js, lc, out, precision="fp64")
    api.run(js, lc, out32, precision="fp32")
    assert rel_l2(out, ref) <= 1e-10
    assert rel_l2(out32, ref) <= 1e-4


@pytest.mark.parametrize("Nx,Ny", [(97, 20), (20, 89), (26, 39), (1, 31), (31, 1), (143, 6)])
@pytest.mark.parametrize("NA", [0.1, 0.45])
def test_focus(gpu, Nx, Ny, NA):
    from nemaktis_gb300.microscope import OpticalFields
    rng = np.random.default_rng(Nx + Ny)
    q = np.array([[0.0, 0.0], [0.1, -0.06]])
    of = OpticalFields(wavelengths=[0.5, 0.6], max_NA_objective=0.5, mesh_dimensions=(Nx, Ny),
                       mesh_lengths=(0.25 * (Nx - 1) or 0.25, 0.25 * (Ny - 1) or 0.25), wavevectors=q)
    shape = (2, 2, 4, Ny, Nx)
    of.vals = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    of.update_NA_objective(NA)
    of.focus_fields(1.7)
    dx, dy = (micrograph.spacing(0.25 * (n - 1) or 0.25, n) for n in (Nx, Ny))
    ref = micrograph.focus_fields(of._vals, [0.5, 0.6], 1.0, q, Nx, Ny, dx, dy, NA, 0.0, 1.7)
    got = of.focused_vals
    scale = np.linalg.norm(of._vals)
    assert np.linalg.norm(got - ref) <= 1e-12 * scale
