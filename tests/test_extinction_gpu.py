"""Spectra between crossed polarisers at oblique angles: dark pixels keep their digits and none is negative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def jones(angle):
    a = np.deg2rad(np.longdouble(angle))
    c, s = np.cos(a), np.sin(a)
    return np.array([[c * c, c * s], [c * s, s * s]], np.clongdouble)


@pytest.mark.parametrize("angle", [17.188, -63.0, 0.0, 90.0])
@pytest.mark.parametrize("noise", [0.0, 1e-9, 1e-6, 1e-2])
def test_crossed_polarisers(gpu, angle, noise):
    """Nearly isotropic fields, polariser at `angle`, analyser crossed. Reference: the Jones product of the focused
    fields in extended precision. Allowed is an error of 32 eps |T| in the Jones entries (two products of 2x2
    matrices whose entries are themselves rounded, the angles' conversion to radians among it)."""
    from nemaktis_gb300.microscope import FieldViewer, OpticalFields
    Nx, Ny = 20, 17
    of = OpticalFields(wavelengths=[0.5, 0.6], max_NA_objective=0.4, max_NA_condenser=0.0, N_radial_wavevectors=1,
                       mesh_lengths=(0.2 * (Nx - 1), 0.25 * (Ny - 1)), mesh_dimensions=(Nx, Ny), n_out=1.0, zfoc_NA_corr=0.0)
    rng = np.random.default_rng(3)
    vals = np.zeros((2, 1, 4, Ny, Nx), complex)
    vals[:, :, 0] = vals[:, :, 3] = np.exp(0.7j)
    of.vals = vals + noise * (rng.normal(size=vals.shape) + 1j * rng.normal(size=vals.shape))
    fv = FieldViewer(of)
    fv.polariser = fv.analyser = True
    fv.polariser_angle, fv.analyser_angle = angle, angle + 90.0
    fv.NA_condenser = 0.0
    fv.update_image()
    got = fv._q_averaged_specter
    F = of.focused_vals.astype(np.clongdouble)[:, 0]  # (l, 2 i + j, y, x): T[j][i]
    T = np.stack([np.stack([F[:, 0], F[:, 2]], -1), np.stack([F[:, 1], F[:, 3]], -1)], -2)
    Y = jones(angle + 90.0) @ T @ jones(angle)
    ref = (0.5 * (np.abs(Y) ** 2).sum((-1, -2))).transpose(1, 2, 0)
    delta = 32 * np.finfo(float).eps * np.sqrt((np.abs(T) ** 2).sum((-1, -2))).transpose(1, 2, 0)
    assert got.shape == ref.shape
    assert got.min() >= 0
    assert (np.abs(got - ref) <= delta * np.sqrt(2 * ref) + 0.5 * delta**2 + 8 * np.finfo(float).eps * ref).all()
