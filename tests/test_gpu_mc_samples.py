"""The batch path's Monte-Carlo models at the edges of the samples a lane counts (4 lanes a pixel: 16, 20, 24 and 32
samples; 8 lanes: 16) against the oracle: the same voxels, values within float32 rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz, nv", [(64, n) for n in (1, 3, 16, 17, 63, 64, 65, 80, 81, 96, 97, 127, 128, 129)] +
                         [(120, n) for n in (1, 16, 17, 100, 128, 129)])
@pytest.mark.parametrize("dv", [5.0, -5.0])
def test_batch_models_per_sample_count(gpu_lib, oracle_lib, nz, nv, dv):
    from bbarolo2_gb300 import _lib, configs, engine
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galmod import ring_rows_batch
    par = Params(CDENS=10, ISEED=1, LTYPE=1, NV=nv, galmodtype="MC")
    cube = Cube.empty(45, 41, nz, [-10. / 3600., 10. / 3600., dv], beam=30. / 3600., par=par,
                      crpix=[23., 21., nz / 2 + 1.], crval=[60., 0., 1000.], cunit=("deg", "deg", "km/s"))
    _, rings = configs.classic64(galmodtype="MC")
    rings.xpos[:], rings.ypos[:] = 22., 20.
    rings.z0[:] = 8.
    dm = engine.DiskModel(cube)
    st = dm.setup
    like = engine.BatchLikelihood(dm, np.ones(cube.array.shape, np.float32), None, maskmode=0, sigma=1.0)
    rows = ring_rows_batch([rings] * 3)
    rows[1, 4, 2] += 7.
    rows[2, 12] += 3.0
    sr, nvs, descs, boxes = like.prepare(rows, rings, seed=3)
    assert int(np.max(nvs)) == nv
    like.run(sr, nvs, descs)
    for k in range(3):
        blo, bhi = boxes[k]
        by, bx = bhi[1] - blo[1], bhi[0] - blo[0]
        got = np.zeros((by, bx, st.nsubs), np.float32)
        dm.ctx.check(dm.ctx.L.bbgpu_eval_model(dm.ctx.h, k, 0, _lib.ptr(got), by, bx, st.nsubs))
        ref = np.zeros((by, bx, st.nsubs))
        oracle_lib.galmod_mc(ref, sr[k], 0, sr.shape[2], 3, st.radsep, nvs[k], st.cdens, st.cmode, st.pixarea,
                             st.cdelt[0], st.cdelt[1], st.crota2, blo[0], blo[1], bhi[0], bhi[1], st.ltype,
                             st.sig_instr, st.axtyp, st.velsys, st.lfreq0, st.crval3, st.cdelt3, st.crpix3, st.relint,
                             st.cd2i)
        assert np.array_equal(got != 0, ref != 0), k
        np.testing.assert_allclose(got, ref, rtol=1e-6, atol=0)
