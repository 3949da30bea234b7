"""The device memory that the stand-alone calls keep: 1 GB at most for the calls of whole cubes, and nothing once
``release_scratch`` has given it back; the next call's result is the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_scratch_is_bounded_and_given_back(gpu_lib):
    import torch
    from bbarolo2_gb300 import configs, engine
    torch.zeros(1, device="cuda")
    cube, rings = configs.classic64()
    dm = engine.DiskModel(cube)
    g = np.random.default_rng(0)
    small = g.random((3, 40, 50))
    first = dm.convolve_planes(small)
    model = dm.array(rings)                                  # (the context's own buffers are there)
    dm.ctx.release_scratch()
    start = _free()
    big = np.zeros((32, 1500, 1500))                         # (16 bytes a voxel: 1.15 GB of scratch)
    big[3, 700, 800] = 1.
    out = dm.convolve_planes(big)
    assert out[3, 700, 800] == np.float32(dm.cfield.max())
    assert start - _free() <= 64 * MB                        # (more than it may keep: given back at its end)
    medium = np.zeros((32, 1100, 1100))                      # (0.6 GB: kept)
    dm.convolve_planes(medium)
    kept = start - _free()
    assert 500 * MB <= kept <= 1100 * MB
    assert np.array_equal(dm.convolve_planes(small), first)
    dm.ctx.release_scratch()
    assert start - _free() <= 64 * MB
    assert np.array_equal(dm.convolve_planes(small), first)
    assert np.array_equal(dm.array(rings), model)
