"""The ANALYTIC batch kernels at the sizes where their tiles and lists can go wrong: boxes that end inside a tile, from
one channel to more than a 4 x 4 tile holds, lines wider than a warp, thick layers of many heights, members of
different boxes. Against the float64 oracle, within the float32 path's bound of 1e-5 of the peak."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nx, ny, nz, channel width (km/s), scale height (arcsec), members
CASES = [(33, 29, 5, 60., 0., 3), (41, 64, 33, 15., 0., 1), (50, 37, 130, 2., 0., 17), (24, 21, 900, 0.5, 0., 2),
         (33, 31, 40, 12., 6., 2), (48, 45, 90, 4., 60., 3), (21, 40, 300, 1., 25., 1)]


@pytest.mark.parametrize("nx,ny,nz,dv,z0,nb", CASES)
def test_tiles(gpu_lib, oracle_lib, nx, ny, nz, dv, z0, nb):
    from bbarolo2_gb300 import _lib, engine
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galmod import ring_rows_batch
    from bbarolo2_gb300.rings import Rings
    par = Params(CDENS=10, ISEED=1, LTYPE=1, galmodtype="ANALYTIC")
    cube = Cube.empty(nx, ny, nz, [-10. / 3600., 10. / 3600., dv], beam=30. / 3600., par=par,
                      crpix=[nx / 2., ny / 2., nz / 2.], crval=[60., 0., 1000.], cunit=("deg", "deg", "km/s"))
    r = np.arange(10., 5. * min(nx, ny) - 20., 20.)
    rings = Rings().setRings(radii=r, xpos=nx / 2. - 3.3, ypos=ny / 2. + 1.7, vsys=1000., vrot=120., vdisp=9., inc=63.,
                             phi=130., z0=z0, dens=np.exp(-r / 60.))
    dm = engine.DiskModel(cube)
    st = dm.setup
    L = engine.BatchLikelihood(dm, np.ones(cube.array.shape, np.float32), None, maskmode=0, sigma=1.0)
    rows = ring_rows_batch([rings] * nb)
    rows[1:, 1:3] += 0.37 * np.arange(nb - 1)[:, None, None]             # (the centre: other boxes)
    rows[1:, 13] += 21. * np.arange(1, nb)[:, None]
    sr, nv, descs, boxes = L.prepare(rows, rings, seed=1)
    L.run(sr, nv, descs, galmodtype="ANALYTIC")
    for k in sorted({0, nb // 2, nb - 1}):
        blo, bhi = boxes[k]
        got = np.zeros((bhi[1] - blo[1], bhi[0] - blo[0], nz), np.float32)
        dm.ctx.check(dm.ctx.L.bbgpu_eval_model(dm.ctx.h, k, 0, _lib.ptr(got), *got.shape))
        ref = np.zeros(got.shape)
        oracle_lib.galmod_analytic(ref, sr[k], 0, sr.shape[2], st.radsep, st.cdens, st.pixarea, st.cdelt[0],
                                   st.cdelt[1], st.crota2, blo[0], blo[1], bhi[0], bhi[1], st.ltype, st.sig_instr,
                                   st._vedges_lines, st.relint, st.cd2i, 1 if z0 == 0 else 1024, st.axtyp, st.velsys,
                                   st.lfreq0, st.crval3, st.cdelt3, st.crpix3, st._chmin, None, st.zstep)
        assert ref.max() > 0
        np.testing.assert_allclose(got, ref, rtol=0, atol=1e-5 * ref.max())
