"""The beam convolution with empty rows of the staged tile left out, against the float64 oracle: kernels of one row and
of one column, widths with even and odd padding, 16- and 32-channel blocks, channels copied 16 and 4 bytes at a time,
sides one off the tiles, planes with bands of zeros, lone pixels and nothing at all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ky, kx", [(1, 1), (1, 7), (9, 1), (3, 3), (15, 15), (11, 25), (31, 31)])
@pytest.mark.parametrize("nz, ny, nx", [(1, 17, 33), (16, 33, 15), (41, 47, 50), (64, 32, 16), (75, 31, 49)])
def test_convolution_of_sparse_planes(gpu_lib, oracle_lib, ky, kx, nz, ny, nx):
    """Error against float64: a rounding of each input and each tap and one of every sum, ky kx + 4 of 2^-24 in all,
    of the same sum with the absolute values."""
    from bbarolo2_gb300 import _lib, configs, engine
    cube, _ = configs.classic64()
    dm = engine.DiskModel(cube)
    g = np.random.default_rng(100 * ky + kx + nz)
    k = np.ascontiguousarray(g.normal(size=(ky, kx)))
    dm.ctx.check(dm.ctx.L.bbgpu_set_kernel(dm.ctx.h, _lib.ptr(k), ky, kx))
    a = g.normal(size=(nz, ny, nx))
    a[:, ny // 3:ny // 2] = 0.
    a[: nz // 2, :, nx // 2:] = 0.
    a[nz // 3] = 0.
    a[nz // 3, ny - 1, nx - 1] = 1.
    a[nz - 1] = 0.
    got = dm.convolve_planes(a)
    want = oracle_lib.conv_same(a, k, 1.0, threshold=False)
    size = oracle_lib.conv_same(np.abs(a), np.abs(k), 1.0, threshold=False)
    assert np.all(np.abs(got - want) <= (ky * kx + 4) * 2. ** -24 * size)
    assert not np.any(got[nz - 1])
