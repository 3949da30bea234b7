"""The float32 normal equations of the flux normalisation at the edges of their blocks of four rings and of their tiles of
128 pixels: the batch's profile against the solve of the float64 system of the same rings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# float32 maps: errors of 2^-23 of the peak of a map, times cond(A), below 10 for rings a beam apart
RTOL = 1e-6


@pytest.mark.parametrize("nx, ny, nr", [(21, 17, 1), (21, 17, 2), (23, 17, 3), (21, 17, 4), (64, 64, 5), (64, 61, 6),
                                        (63, 64, 7), (64, 64, 8), (64, 64, 15), (128, 127, 30), (128, 128, 31)])
def test_batch_profile_sizes(gpu_lib, nx, ny, nr):
    from bbarolo2_gb300 import engine, profile as P
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galmod import ring_rows_batch
    from bbarolo2_gb300.rings import Rings
    par = Params(CDENS=10, ISEED=1, LTYPE=2, galmodtype="ANALYTIC")
    cube = Cube.empty(nx, ny, 24, [-10. / 3600., 10. / 3600., 20.], beam=20. / 3600., par=par,
                      crpix=[(nx + 1) / 2., (ny + 1) / 2., 12.5], crval=[60., 0., 1000.],
                      cunit=("deg", "deg", "km/s"))
    rmax = 10. * 0.45 * min(nx, ny)
    r = (np.arange(nr) + 0.5) * rmax / nr
    rings = Rings().setRings(radii=r, xpos=(nx - 1) / 2., ypos=(ny - 1) / 2., vsys=1000., vrot=100., vdisp=20.,
                             inc=50., phi=40., z0=8., dens=np.exp(-r / rmax))
    dm = engine.DiskModel(cube, galmodtype="ANALYTIC")
    g = np.random.default_rng(nr)
    data = np.asarray(dm.array(rings), np.float32)
    data += g.normal(0., 0.01 * data.max(), data.shape).astype(np.float32)
    like = engine.BatchLikelihood(dm, data, np.ones(data.shape, bool), maskmode=2, sigma=0.01 * float(data.max()))
    mom0, rms, ok = like.data_maps()
    like.set_profile(rings, mom0, rms, ok, smooth=0.3, corr=4.0, beam_arcsec=20.)
    rows = ring_rows_batch([rings] * 3)
    rows[1, 12] += 2.
    rows[2, 13, -1] += 5.
    ll = like.evaluate(rows, rings, seed=1)
    x, st = like.last_profile()
    assert not np.any(np.asarray(st) & 1)
    for k in (1, 2):                                         # (a member's profile does not depend on the batch)
        assert like.evaluate(rows[k:k + 1], rings, seed=1)[0] == ll[k]
    want = P.deconvolved_profile(dm, rings, like.likebox, mom0, rms, ok, 0.3, beam_arcsec=20., corr=4.0)
    np.testing.assert_allclose(x[0, :nr], want, rtol=RTOL, atol=RTOL * np.abs(want).max())
