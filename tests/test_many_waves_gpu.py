"""More (wavelength, q) waves than a grid has places along its second dimension (65535): the screen of a sample
propagated wavelength by wavelength, and the micrograph's focus."""
import numpy as np
import pytest

import oracle
from nemaktis_gb300 import api
from tests.helpers import case, rel_l2

pytestmark = pytest.mark.gpu

NQ = 4100


def wavevectors():
    return np.random.default_rng(1).uniform(-0.2, 0.2, (NQ, 2))


def test_screen(gpu):
    js, lc, shape = case((4, 4, 2), wavelengths=np.linspace(0.4, 0.7, 8), q=wavevectors(), seed=2)
    ref, out = np.zeros(shape, np.complex128), np.zeros(shape, np.complex128)
    oracle.run_backend_without_mask(js, lc, ref)
    api.run(js, lc, out, precision="fp64", groups_per_pass=1)
    assert rel_l2(out, ref) <= 1e-10  # as for the parity tests


def test_focus(gpu):
    from nemaktis_gb300.microscope import OpticalFields
    wl = np.linspace(0.4, 0.7, 16)
    kw = dict(max_NA_objective=0.5, max_NA_condenser=0.3, N_radial_wavevectors=2, mesh_lengths=(0.6, 0.9), mesh_dimensions=(4, 4),
              n_out=1.0, zfoc_NA_corr=0.0, wavevectors=wavevectors())
    rng = np.random.default_rng(3)
    vals = rng.normal(size=(16, NQ, 4, 4, 4)) + 1j * rng.normal(size=(16, NQ, 4, 4, 4))
    of = OpticalFields(wavelengths=wl, **kw)
    of.vals = vals
    of.focus_fields(1.5)
    for k in (0, 7, 15):
        one = OpticalFields(wavelengths=[wl[k]], **kw)
        one.vals = vals[k:k + 1]
        one.focus_fields(1.5)
        np.testing.assert_array_equal(of.focused_vals[k], one.focused_vals[0])
