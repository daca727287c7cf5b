"""Mask weights for formulas whose parts have none, one, two and three variables: the parts of one variable are
taken from tables, the rest is evaluated point by point. A bisection stops within 1e-3 of a cell and its steps
are the oracle's, so the weights agree to the rounding of the formula (1e-12)."""

import ctypes

import numpy as np
import pytest

import oracle
from nemaktis_gb300 import _lib, workloads
from oracle import expr

FORMULAS = ["0.7-z", "x+0.013", "z^2*0+1", "2.2^2-x^2-y^2-(z-0.1)^2", "x*z-y*z+0.05", "min(1.1-abs(z),2-x^2,2-y)",
            "x>y ? 0.5-z^3 : z-x*y*0.2", "avg(x,y,z,0.1)", "exp(x*0.1)*cos(z*y)-0.4", "-(x-0.1)^2/(1+y^2)+z^2-0.3",
            "(z<0.4)&&(x<0.2) ? 1 : -1", "sqrt(x)-z"]


@pytest.mark.parametrize("dims", [(1, 1, 2), (7, 5, 9), (5, 3, 1), (3, 8, 2)])
@pytest.mark.parametrize("formula", FORMULAS)
def test_mask_weights_of_formulas(formula, dims):
    lib = _lib.load()
    d = (0.31, 0.29, 0.23)
    js = workloads.settings_json(dims, d, [0.6], [0.0, 0.0])
    ax = [(np.arange(n) - 0.5 * (n - 1)) * h for n, h in zip(dims, d)]
    vals = np.empty(dims[::-1])
    for k, z in enumerate(ax[2]):
        for j, y in enumerate(ax[1]):
            for i, x in enumerate(ax[0]):
                with np.errstate(all="ignore"):
                    vals[k, j, i] = expr.evaluate(formula, x=x, y=y, z=z)
    n = vals.size
    m = np.zeros(n, np.uint8)
    w = np.zeros(2 * (n - dims[0] * dims[1]) + 1)
    assert lib.nbpm_mask_weights(js.encode(), formula.encode(), vals.ctypes.data, n, m.ctypes.data,
                                 w.ctypes.data) == 0
    with np.errstate(all="ignore"):
        m_ref, w_ref = oracle.mask_interp_weights(vals, formula, dims, d)
    assert np.array_equal(m, m_ref.ravel())
    assert np.allclose(w[:-1], w_ref.ravel(), rtol=0, atol=1e-12, equal_nan=True)
