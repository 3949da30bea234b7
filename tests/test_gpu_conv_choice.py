"""The batch convolution's choice between float32 and tf32x3: the faster of the two as they run, by the times that it
reports; and the float32 kernel that is timed against the tensor cores gives the bits of the one that leaves rows of
zeros out (option 4 = 0)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PIX = 8.0


def _problem(nx, nz, bmaj, bmin, nb, model, gradient=False):
    """A thick disk that fills the cube and the band, nb ring sets about it; noise as the data."""
    from bbarolo2_gb300 import engine
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galmod import ring_rows_batch
    from bbarolo2_gb300.rings import Rings
    nr = nx // 4 - 1
    rad = (0.5 + np.arange(nr)) * 2.0 * PIX
    vrot = 190. * (2 / math.pi) * np.arctan(rad / (0.1 * rad[-1]))
    rings = Rings().setRings(radii=rad, xpos=(nx - 1) / 2., ypos=(nx - 1) / 2., vsys=1000., vrot=vrot,
                             vdisp=np.linspace(12., 7., nr), inc=np.full(nr, 60.), phi=np.full(nr, 40.),
                             z0=np.full(nr, 0.8 * PIX), dens=0.8 * np.exp(-rad / (0.3 * rad[-1])))
    dv = 2. * (190. * math.sin(math.radians(60.)) + 40.) / (0.8 * nz)
    par = Params(CDENS=10, ISEED=1, LTYPE=2, galmodtype=model)
    cube = Cube.empty(nx, nx, nz, [-PIX / 3600., PIX / 3600., dv], beam=[bmaj * PIX / 3600., bmin * PIX / 3600., 30.],
                      par=par, crpix=[nx / 2. + 0.5, nx / 2. + 0.5, nz // 2 + 1.], crval=[60., 0., 1000.],
                      cunit=("deg", "deg", "km/s"))
    dm = engine.DiskModel(cube, galmodtype=model)
    g = np.random.default_rng(nx + nz)
    data = g.standard_normal((nz, nx, nx), dtype=np.float32)
    L = engine.BatchLikelihood(dm, data, np.ones(data.shape, bool), maskmode=2, sigma=1.)
    rows = ring_rows_batch([rings] * nb)
    if gradient:
        for k in range(1, nb):
            rows[k, 4, (k - 1) % nr] += 2.
    else:
        rows[:, 4] += g.uniform(-5., 5., (nb, nr))
    return dm, L, rings, rows


# (shapes at which the two variants take about the same time)
@pytest.mark.parametrize("nx, nz, bmaj, bmin, nb", [(96, 76, 3.5, 3.5, 3), (120, 72, 4.0, 2.8, 2), (51, 76, 3.0, 3.0, 45),
                                                    (104, 48, 3.5, 3.5, 101), (144, 40, 4.1, 3.5, 60),
                                                    (88, 108, 3.5, 2.9, 7), (168, 92, 2.6, 1.9, 5)])
def test_choice_is_the_faster(gpu_lib, nx, nz, bmaj, bmin, nb):
    from bbarolo2_gb300 import _lib
    dm, L, rings, rows = _problem(nx, nz, bmaj, bmin, nb, "ANALYTIC")
    a = L.evaluate(rows, rings, seed=1)
    used, ms = dm.ctx.conv_variant()
    assert set(ms) == {"f32", "tf32x3"} and all(v > 0 for v in ms.values()), ms
    assert used == (_lib.CONV_TF32X3 if ms["tf32x3"] < ms["f32"] else _lib.CONV_F32), (used, ms)
    np.testing.assert_array_equal(a, L.evaluate(rows, rings, seed=1))


# (small batches: float32 by a third and more; 32 and 16 channels a block; own tiles and, in a gradient, shared ones)
@pytest.mark.parametrize("nx, nz, nb, model, gradient", [(48, 64, 1, "ANALYTIC", False), (49, 36, 2, "ANALYTIC", False),
                                                        (50, 64, 3, "MC", True), (45, 44, 3, "MC", True)])
def test_float32_kernels_agree(gpu_lib, nx, nz, nb, model, gradient):
    from bbarolo2_gb300 import _lib
    dm, L, rings, rows = _problem(nx, nz, 3.0, 2.5, nb, model, gradient)
    a = L.evaluate(rows, rings, seed=1)
    used, ms = dm.ctx.conv_variant()
    assert used == _lib.CONV_F32, (used, ms)
    dm.ctx.set_option(4, 0)
    b = L.evaluate(rows, rings, seed=1)
    dm.ctx.set_option(4, -1)
    assert np.all(np.isfinite(a))
    np.testing.assert_array_equal(a, b)
