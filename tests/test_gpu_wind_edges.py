"""GALWIND clouds on the edge between two pixels, as the C library's sine and cosine place them: GalWindMC against the
oracle, which takes them from there. XPOS is such that the pixel coordinate of one cloud is 1/2 exactly, to the last bit:
a position an ulp lower belongs to pixel 0."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("shim") / "libwindshim.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-o", out,
                    os.path.join(HERE, "host", "wind_clouds_shim.cpp"),
                    os.path.join(os.path.dirname(HERE), "bbarolo2_gb300", "csrc", "host_setup.cpp")], check=True)
    return C.CDLL(out)


def _offsets(L, gw, seed):
    """The clouds' pixel offsets from XPOS (bbarolo/galmod.py:571-574), each operation rounded once."""
    st, p = gw.setup, lambda a: None if a is None else a.ctypes.data_as(C.c_void_p)
    args = [C.c_uint64(seed), p(gw.sr), C.c_int(gw.sr.shape[1]), C.c_int(0), C.c_int(gw.sr.shape[1]),
            C.c_double(gw.sep), p(gw.nv), C.c_double(st.cdens), C.c_int(1), C.c_double(st.pixarea),
            C.c_double(st.sig_instr), C.c_double(st.crota2)]
    n = np.zeros(4, np.int64)
    assert L.wind_clouds_dump(*args, p(n), *[None] * 8) == 0
    sh, of, geo = np.zeros((n[0], 12)), np.zeros(n[1], np.int32), np.zeros((n[1], 5))
    assert L.wind_clouds_dump(*args, p(n), p(sh), p(of), p(geo), *[None] * 4) == 0
    sinc, cinc, spa, cpa = sh[of, 5:9].T
    rad, caz, saz, sphi, cphi = geo.T
    x, y = rad * sphi * caz, rad * sphi * saz * cinc - rad * cphi * sinc
    return (x * spa - y * cpa) / st.cdelt[0]


def test_clouds_on_pixel_edges(gpu_lib, oracle_lib, shim):
    from bbarolo2_gb300.cube import Cube, Params
    from bbarolo2_gb300.galwind import GalWindMC, GalWindPars
    cube = Cube.empty(40, 24, 32, [-4. / 3600., 4. / 3600., 20.], par=Params(), crpix=[20.5, 12.5, 16.5],
                      crval=[60., 0., 0.], cunit=("deg", "deg", "km/s"))
    par = GalWindPars(xpos=20., ypos=11.7, vsys=5., inc=58., phi=37., conelen=64., nlayers=3, vwind=250., vdisp=25.,
                      dens=10., openang=70., cdens=2., nv=10, iseed=5)
    gw = GalWindMC(cube, par, threads=1)
    st = gw.setup
    q = _offsets(shim, gw, 5)
    assert q.size * 13 > 20000                               # (the streams are followed on the device)
    xpos = 0.5 - q
    good = np.flatnonzero((xpos + q == 0.5) & (np.abs(q) > 4) & (np.abs(q) < 12))
    assert good.size > 100
    for i in good[:: good.size // 60][:60]:
        gw.sr[8] = xpos[i]
        mod = gw.model()
        ref = oracle_lib.galmod_wind(np.zeros((24, 40, 32)), gw.sr, 0, gw.sr.shape[1], 5, gw.sep, gw.nv, st.cdens, 1,
                                     st.pixarea, st.cdelt[0], st.cdelt[1], st.crota2, 0, 0, 40, 24, st.sig_instr,
                                     st.axtyp, st.velsys, st.lfreq0, st.crval3, st.cdelt3, st.crpix3, st.relint,
                                     st.cd2i).transpose(2, 0, 1)
        assert np.array_equal(mod != 0, ref != 0)
        np.testing.assert_allclose(mod, ref, rtol=1e-9, atol=0)
