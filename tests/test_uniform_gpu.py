"""A uniform field passes a uniform director along z with no more change than rounding: its phase is zero and the line
solves answer a constant with itself, so that what their coefficients' rounding takes of it, the same at every point of
every slab, adds up along the propagation. 200 slabs against one, FP64, weak coupling. A solve repeats the rounding
of five factors of at most a quarter (2^-55 each, signs by chance): 400 solves x 2^-55 x sqrt(5) = 2.5e-14. With 1/beta
itself among them, rounded to 2^-53, droplets of 64 slabs were off by a third more."""
import numpy as np
import pytest

from nemaktis_gb300 import api
from tests.helpers import case

pytestmark = pytest.mark.gpu


def fields(dims, index, wavelength, cfg):
    lc = np.zeros((dims[2], dims[1], dims[0], 3))
    lc[..., 2] = 1
    js, _, shape = case(dims, lc=lc, no=index, ne="1.75", wavelengths=(wavelength,))
    E = np.zeros(shape, np.complex128)
    api.run(js, lc, E, precision="fp64", solve_config=cfg)
    return E[0, 0, [0, 3]]  # each polarisation's own component


@pytest.mark.parametrize("index,wavelength", [("1.55", 0.6), ("1.5", 0.5), ("1.62", 0.45), ("1.4", 0.7)])
@pytest.mark.parametrize("dims,cfg", [((128, 128), "xc:M=4:KS=1;yx:M=4:KS=1"), ((256, 20), "xc:M=8:KS=2;yx:M=2:KS=2"),
                                      ((300, 12), "xw:M=8:KS=2:W=2;yx:M=2:KS=2"), ((12, 300), "xc:M=2:KS=1;yx:M=8:KS=1:W=2")])
def test_uniform_field_is_kept(gpu, dims, cfg, index, wavelength):
    one, many = fields((*dims, 2), index, wavelength, cfg), fields((*dims, 201), index, wavelength, cfg)
    assert np.abs(many / one - 1).max() <= 2.5e-14
