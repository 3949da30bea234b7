"""GALWIND's streams followed on the device (``csrc/galwind.cu``, k_ws_*): the models of GalWindMC against the oracle's
``_galmod_wind`` over the same chunks, at the lengths where the device's blocks and rounds can go wrong: one chunk and
many, the fewest and the most draws a cloud, a stream of more words than a round takes, and one draw a cloud more than
the device follows (parsed on the host). One misplaced word would move every later cloud of its chunk.

Values: a deposit is rounded to 2^-62 of twice the total flux at most, the deposits of a model are nearly equal, so a
voxel of one deposit is off by at most the model's number of deposits x 2^-61 of its value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# velocity samples, clouds per pixel, chunks, cone length (pixels)
CASES = [(20, 0.3, 1, 6.), (20, 4., 3, 20.), (1, 40., 5, 30.), (7, 11., 16, 33.), (125, 9., 2, 30.), (126, 0.5, 2, 12.),
         (125, 180., 1, 28.)]


@pytest.mark.parametrize("nv,cdens,threads,cone", CASES)
def test_stream(gpu_lib, oracle_lib, nv, cdens, threads, cone):
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galwind import GalWindMC, GalWindPars
    cube = Cube.empty(61, 57, 40, [-4. / 3600., 4. / 3600., 16.], par=Params(), crpix=[31., 29., 20.5],
                      crval=[60., 0., 0.], cunit=("deg", "deg", "km/s"))
    par = GalWindPars(xpos=30.2, ypos=27.6, vsys=5., inc=58., phi=37., conelen=4. * cone, nlayers=3, vwind=250.,
                      vdisp=25., dens=10., openang=70., cdens=cdens, nv=nv, iseed=11)
    gw = GalWindMC(cube, par, threads=threads)
    mod = gw.model()
    st = gw.setup
    ref = np.zeros((cube.DimY(), cube.DimX(), cube.DimZ()))
    for k, ch in enumerate(gw.chunks()):
        ref += oracle_lib.galmod_wind(np.zeros_like(ref), gw.sr, int(ch[0]), int(ch[-1]) + 1,
                                      (11 + 7919 * k) & 0xFFFFFFFF, gw.sep, gw.nv, st.cdens, 1, st.pixarea,
                                      st.cdelt[0], st.cdelt[1], st.crota2, 0, 0, cube.DimX(), cube.DimY(),
                                      st.sig_instr, st.axtyp, st.velsys, st.lfreq0, st.crval3, st.cdelt3, st.crpix3,
                                      st.relint, st.cd2i)
    ref = ref.transpose(2, 0, 1)
    nc = np.rint(st.cdens * gw.sr[4] * 2 * np.pi * gw.sr[0] * gw.sep / st.pixarea).sum()
    assert np.array_equal(mod != 0, ref != 0)
    np.testing.assert_allclose(mod, ref, rtol=max(nc * nv * 2. ** -61, 1e-12), atol=0)
