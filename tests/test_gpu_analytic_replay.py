"""ANALYTIC members that are member 0 but for the fluxes (computed from its runs) against the same members computed from
all their samples: equal bit for bit, models and sums. Channels one off the blocks of 32, members one off the groups of
16, sub-rings of their own, a sub-ring without flux."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz, nb", [(1, 10), (31, 10), (32, 17), (33, 18), (64, 34), (100, 12)])
@pytest.mark.parametrize("z0, nr", [(12., 8), (4., 1), (25., 3), (6., 90)])
def test_replayed_members(gpu_lib, nz, nb, z0, nr):
    from bbarolo2_gb300 import _lib, configs, engine
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galmod import ring_rows_batch
    from bbarolo2_gb300.rings import Rings
    par = Params(CDENS=10, ISEED=1, LTYPE=2, galmodtype="ANALYTIC")
    cube = Cube.empty(37, 41, nz, [-10. / 3600., 10. / 3600., 5.], beam=30. / 3600., par=par,
                      crpix=[19., 21., nz / 2 + 1.], crval=[60., 0., 1000.], cunit=("deg", "deg", "km/s"))
    _, rings = configs.classic64(galmodtype="ANALYTIC")
    if nr > rings.nr:                                        # (amplitudes that take more than 48 KB of shared memory)
        r = 4. + 8. * np.arange(nr)
        rings = Rings().setRings(radii=r, vsys=1000., vrot=150. * (1 - np.exp(-r / 40.)), vdisp=10., inc=55., phi=45.,
                                 dens=np.exp(-r / 60.))
    rings = rings.subset(list(range(nr)))
    rings.xpos[:], rings.ypos[:], rings.z0[:] = 18., 20., z0
    dm = engine.DiskModel(cube)
    like = engine.BatchLikelihood(dm, np.ones(cube.array.shape, np.float32), None, maskmode=0, sigma=1.0)
    g = np.random.default_rng(nb)
    rows = np.repeat(ring_rows_batch([rings]), nb, axis=0)
    rows[1:, 10] *= g.uniform(0.2, 5., (nb - 1, nr))         # (densities)
    rows[3, 10, nr - 1] = 0.
    if nr > 3:
        for k in range(4, nb):
            rows[k, 12 if k % 2 else 13, k % nr] += 3.       # (INC or PA of one ring)
    sr, nv, descs, boxes = like.prepare(rows, rings, seed=1)
    assert nr <= 8 or sr.shape[2] > 75
    out = {}
    try:
        for share in (0, 1):
            dm.ctx.set_option(_lib.OPT_SHARE, share)
            ss, _ = like.run(sr, nv, descs)
            ms = []
            for k in range(nb):
                blo, bhi = boxes[k]
                got = np.zeros((bhi[1] - blo[1], bhi[0] - blo[0], nz), np.float32)
                dm.ctx.check(dm.ctx.L.bbgpu_eval_model(dm.ctx.h, k, 0, _lib.ptr(got), got.shape[0], got.shape[1], nz))
                ms.append(got)
            out[share] = ss, ms
            if share:
                assert dm.ctx.shared_members()[3] >= nb - 2
    finally:
        dm.ctx.set_option(_lib.OPT_SHARE, 1)
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)
    assert any(m.any() for m in out[1][1])
