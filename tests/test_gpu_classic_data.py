"""The data that a CLASSIC evaluation is compared with: those of the grid in hand and of the call."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(seed):
    from bbarolo2_gb300 import classic, configs
    from golden.cases import galfit_par
    cube, rings = configs.classic64()
    g = np.random.default_rng(seed)
    data = g.normal(0., 0.05, cube.array.shape).astype(np.float32)
    data[20:44] += 0.2
    cube.array = data
    par = galfit_par()
    par.NORM, par.NORMALCUBE = "LOCAL", False
    return classic.ClassicFit(cube, rings, par, 0.05, g.random(data.shape) < 0.7)


def test_data_of_another_grid_are_refused(gpu_lib):
    from bbarolo2_gb300 import _lib
    fit = _fit(1)
    fit.run(rings=[])
    st, ctx = fit.model.setup, fit.ctx
    sr, nv = st.subrings(fit.inr)
    sr, nv = np.ascontiguousarray(sr, np.float64), np.ascontiguousarray(nv, np.int64)

    def residual():
        out = np.zeros(1)
        rc = ctx.L.bbgpu_classic_residual(ctx.h, _lib.ptr(sr), sr.shape[1], ctypes.c_uint64(1), _lib.ptr(nv), 0, 0, 64,
                                          64, None, 0, 0, 1.0, 32., 32., 45., 60., 0., 10., 1., 0, 2, 0.05, 1., 0,
                                          _lib.ptr(out))
        return rc, out[0]

    rc, value = residual()
    assert rc == _lib.OK and np.isfinite(value)
    grid = fit.model._grid()
    edges = np.asarray(st._vedges_lines, float).reshape(-1)
    args = [_lib.ptr(st.cd2i), _lib.ptr(st.lfreq0), _lib.ptr(st.relint), _lib.ptr(edges)]
    ctx.check(ctx.L.bbgpu_set_grid(ctx.h, grid, *args))
    assert residual()[0] == _lib.ERR_STATE                   # (the same grid set anew)
    more = np.concatenate([st.cd2i, st.cd2i])
    wide = np.concatenate([edges, edges[-1] + np.arange(1, st.nsubs + 1) * (edges[-1] - edges[-2])])
    grid.nz = 2 * st.nsubs
    ctx.check(ctx.L.bbgpu_set_grid(ctx.h, grid, _lib.ptr(more), args[1], args[2], _lib.ptr(wide)))
    assert residual()[0] == _lib.ERR_STATE                   # (more channels than the data have)
    fit.model.ctx.check(ctx.L.bbgpu_set_grid(ctx.h, fit.model._grid(), *args))
    fit.run(rings=[])
    rc, again = residual()
    assert rc == _lib.OK and again == value


@pytest.mark.parametrize("change", ["data", "mask", "chan_noise"])
def test_residual_takes_what_it_is_given(gpu_lib, change):
    """Other data, another mask or noise than the last run's: the value of a fit that ran with them."""
    from bbarolo2_gb300 import classic
    a, b = _fit(1), _fit(2)
    if change != "data":
        b.cube.array = a.cube.array
    if change != "mask":
        b.mask_yxz, b.mask2d = a.mask_yxz, a.mask2d
    if change == "chan_noise":
        b.chan_noise = np.linspace(1., 3., 64)
    ring = classic.ring_annulus(a.inr, 4)
    yxz = [np.ascontiguousarray(f.cube.array.transpose(1, 2, 0)) for f in (a, b)]
    for f in (a, b):
        f.par.FTYPE = 1                                      # (the residual that the noise weights)
        f.run(rings=[])
    va, vb = a._residual(ring, yxz[0], 0.05, 0), b._residual(ring, yxz[1], 0.05, 0)
    assert va != vb
    a.mask_yxz, a.chan_noise = b.mask_yxz, b.chan_noise
    assert a._residual(ring, yxz[1], 0.05, 0) == vb


def test_kernel_of_any_layout(gpu_lib):
    """A beam kernel that is not C-contiguous."""
    from bbarolo2_gb300 import classic
    fit = _fit(3)
    k = np.array(fit.model.cfield)
    k[0] *= 0.25                                             # (not its own transpose)
    ring = classic.ring_annulus(fit.inr, 3)
    data = np.ascontiguousarray(fit.cube.array.transpose(1, 2, 0))
    fit.run(rings=[])
    fit.model.cfield = k
    want = fit._residual(ring, data, 0.05, 0)
    fit.model.cfield = np.asfortranarray(k)
    assert fit._residual(ring, data, 0.05, 0) == want
    fit.model.cfield = k.T
    assert fit._residual(ring, data, 0.05, 0) != want
