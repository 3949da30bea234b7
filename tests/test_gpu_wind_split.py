"""The columns handed to the convolution as float-float: with a beam of one tap the convolution returns the pair as it is,
which is within 2^-49 of the deposited sum (the column without a beam): the high word is the sum rounded to 24 bits, the
low word the rest (at most 2^-25) rounded to 24."""
import numpy as np
import pytest

import wind_cases as WC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("separable", [True, False])
def test_pairs_hold_49_bits(gpu_lib, separable):
    from bbarolo2_gb300 import wind
    cube = WC.cube(40, 32, beam=(30.,))
    P = wind.WindPars([60., 140.], [120., 220.], [12., 9.], vrot=[40., 10.], xpos=19.7, ypos=20.4, inc=55., pa=30.,
                      openang=70., openin=10., conelen=150.)
    cols = []
    for hx in (0, 1):
        wm = wind.WindModel(cube, wind.WindCells.resolved(160., 40., 25.), smooth=False).quadrature(200., 10.)
        if hx:
            wm.hx = wm.hy = 1
            wm.kern = np.zeros((3, 3))
            wm.kern[1, 1] = 1.
            wm.kx = wm.ky = np.array([0., 1., 0.])
            wm.separable = separable
        B = wm.boxes(P)
        cols.append([B.column(k, wm.shape) for k in range(wm.cells.ncell)])
    n = 0
    for a, b in zip(*cols):
        at = a != 0
        n += int(at.sum())
        assert np.array_equal(at, b != 0)
        assert np.all(np.abs(b[at] - a[at]) <= 2. ** -49 * (1 + 2. ** -6) * np.abs(a[at]))
    assert n > 10000
