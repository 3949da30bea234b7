"""The calls that build and convolve a model (or build, convolve and compare a CLASSIC ring) in one go against the
separate calls they stand for: the full model box, ragged ones, one pixel, rings of one tile and of many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gtype", ["MC", "ANALYTIC"])
@pytest.mark.parametrize("z0", [0.0, 12.0])
@pytest.mark.parametrize("blo, bhi", [((0, 0), (64, 64)), ((20, 11), (49, 48)), ((32, 32), (33, 33)),
                                      ((0, 60), (64, 64))])
def test_model_cube(gpu_lib, gtype, z0, blo, bhi):
    """The float32 input of the convolution differs from the separate calls' by at most an ulp (the float64 model
    is not rounded twice), so each output by ky kx + 8 rounding errors of its sum of positive terms, and by 1e-12 where
    the cut falls."""
    from bbarolo2_gb300 import configs, engine
    from bbarolo2_gb300.galmod import model_rings
    cube, rings = configs.classic64(galmodtype=gtype)
    rings.z0[:] = z0
    dm = engine.DiskModel(cube, galmodtype=gtype)
    got = dm.array(rings, blo, bhi, final=True)
    mr = model_rings(rings, dm.ringmode, dm.setup.radsep)
    want = dm.convolve(dm.build(mr, blo, bhi, layout="yxz"), "zyx")
    assert got.shape == want.shape
    tol = (dm.cfield.size + 8) * 2. ** -23
    assert np.all(np.abs(got - want) <= tol * np.abs(want) + 1e-12 * dm.scalefactor)
    assert np.array_equal(dm.array(rings, blo, bhi, final=True, layout="yxz"), got.transpose(1, 2, 0))


@pytest.mark.parametrize("ring", [0, 3, 7])
@pytest.mark.parametrize("norm", ["LOCAL", "AZIM", "NONE"])
@pytest.mark.parametrize("xpos, inc", [(32., 55.), (3.5, 20.), (62., 85.)])
def test_classic_residual(gpu_lib, ring, norm, xpos, inc):
    """The same model bit for bit, so the value differs by the order of the residual's sum: 1e-12."""
    from bbarolo2_gb300 import classic, configs
    from bbarolo2_gb300.galfit import _norm
    from golden.cases import galfit_par
    cube, rings = configs.classic64()
    g = np.random.default_rng(ring)
    data = g.normal(0., 0.05, cube.array.shape).astype(np.float32)
    data[20:44] += 0.2
    cube.array = data
    mask = g.random(data.shape) < 0.7
    rings.xpos[:] = xpos
    rings.inc[:] = inc
    par = galfit_par()
    par.NORM, par.NORMALCUBE = norm, False
    fit = classic.ClassicFit(cube, rings, par, 0.05, mask)
    fit.run(rings=[])                                       # (sets the data and the mask)
    dring = classic.ring_annulus(fit.inr, ring)
    data_yxz = np.ascontiguousarray(data.transpose(1, 2, 0))
    got = fit._residual(dring, data_yxz, 0.05, classic.NORMCODE[norm])
    blo, bhi = fit.model.box(dring)
    mod = np.ascontiguousarray(fit.model.array(dring, blo, bhi, final=False, layout="yxz"), np.float64)
    want = _norm(mod, data_yxz, fit.mask_yxz, blo[0], blo[1], xpos - blo[0], 32. - blo[1], 45., inc,
                 dring.radii[0] / fit.pixscale, dring.radii[-1] / fit.pixscale, float(par.WFUNC),
                 classic.SIDECODE.get(par.SIDE, 0), par.FTYPE, fit.chan_noise, 0.05, par.BWEIGHT,
                 classic.NORMCODE[norm], None, None, None, None, None, 0, 0., ctx=fit.ctx)
    assert got == want or abs(got - want) <= 1e-12 * abs(want)
