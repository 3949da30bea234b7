"""Thin ANALYTIC disks whose channels are written 16 bytes at a time (channels a multiple of 4), many samples a pixel,
deposits on both sides of 2^44 units: the models equal, bit for bit, those whose channels are written one at a time
(members as differences from member 0), and the float64 oracle's within the float32 path's 1e-5 of the peak."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [4, 32, 36, 132])
@pytest.mark.parametrize("inc, nx", [(87., 15), (60., 40)])
def test_pixels_by_16_bytes(gpu_lib, oracle_lib, nz, inc, nx):
    from bbarolo2_gb300 import _lib, engine
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galmod import ring_rows_batch
    from bbarolo2_gb300.rings import Rings
    par = Params(CDENS=10, ISEED=1, LTYPE=1, galmodtype="ANALYTIC")
    cube = Cube.empty(nx, nx, nz, [-10. / 3600., 10. / 3600., 400. / nz], beam=30. / 3600., par=par,
                      crpix=[nx / 2., nx / 2., nz / 2.], crval=[60., 0., 1000.], cunit=("deg", "deg", "km/s"))
    r = np.arange(5., 5. * nx, 10.)
    rings = Rings().setRings(radii=r, xpos=nx / 2. - 0.6, ypos=nx / 2. - 0.3, vsys=1000., vrot=120., vdisp=9., inc=inc,
                             phi=35., z0=0., dens=np.exp(-r / (2. * nx / 5.)))
    dm = engine.DiskModel(cube)
    st = dm.setup
    L = engine.BatchLikelihood(dm, np.ones(cube.array.shape, np.float32), None, maskmode=0, sigma=1.0)
    nb = 5
    rows = ring_rows_batch([rings] * nb)
    for k in range(1, nb):
        rows[k, 4, k % rings.nr] += 7.                       # (VROT of one ring)
    sr, nv, descs, boxes = L.prepare(rows, rings, seed=1)
    out = {}
    try:
        for share in (0, 1):
            dm.ctx.set_option(_lib.OPT_SHARE, share)
            L.run(sr, nv, descs, galmodtype="ANALYTIC")
            if share:
                assert dm.ctx.shared_members()[2] == nb - 1
            ms = []
            for k, (blo, bhi) in enumerate(boxes):
                got = np.zeros((bhi[1] - blo[1], bhi[0] - blo[0], nz), np.float32)
                dm.ctx.check(dm.ctx.L.bbgpu_eval_model(dm.ctx.h, k, 0, _lib.ptr(got), *got.shape))
                ms.append(got)
            out[share] = ms
    finally:
        dm.ctx.set_option(_lib.OPT_SHARE, 1)
    for k, (blo, bhi) in enumerate(boxes):
        np.testing.assert_array_equal(out[0][k], out[1][k])
        ref = np.zeros(out[0][k].shape)
        oracle_lib.galmod_analytic(ref, sr[k], 0, sr.shape[2], st.radsep, st.cdens, st.pixarea, st.cdelt[0],
                                   st.cdelt[1], st.crota2, blo[0], blo[1], bhi[0], bhi[1], st.ltype, st.sig_instr,
                                   st._vedges_lines, st.relint, st.cd2i, 1, st.axtyp, st.velsys, st.lfreq0, st.crval3,
                                   st.cdelt3, st.crpix3, st._chmin, None, st.zstep)
        assert ref.max() > 0
        np.testing.assert_allclose(out[0][k], ref, rtol=0, atol=1e-5 * ref.max())
