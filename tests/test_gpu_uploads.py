"""Batches uploaded one after another while earlier runs are still queued: each upload waits for the last one's copies
from the pinned arrays, so that a run never sees the members of the next batch. The values read at the end are the last
batch's, and a batch read after a pile of others is what it is alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gtype", ["ANALYTIC", "MC"])
def test_uploads_behind_runs(gpu_lib, gtype):
    from bbarolo2_gb300 import _lib, configs, engine
    from bbarolo2_gb300.galmod import ring_rows_batch
    cube, rings = configs.classic64(galmodtype=gtype)
    dm = engine.DiskModel(cube, galmodtype=gtype)
    g = np.random.default_rng(3)
    L = engine.BatchLikelihood(dm, g.random(cube.array.shape, dtype=np.float32), None, maskmode=0, sigma=1.0)
    code = _lib.ANALYTIC if gtype == "ANALYTIC" else _lib.MC
    batches = []
    for i, nb in enumerate((48, 2, 40, 1, 64, 7)):           # (more and fewer members, the centre and so the box moving)
        rows = ring_rows_batch([rings] * nb)
        rows[:, 1:3] += g.uniform(-6., 6., (nb, 2, 1))
        rows[:, 4] += g.uniform(-5., 5., (nb, rings.nr))
        batches.append(L.prepare(rows, rings, seed=1))
    ctx = dm.ctx

    def queue(k, runs):
        sr, nv, descs, _ = batches[k]
        ctx.check(ctx.L.bbgpu_eval_upload(ctx.h, code, sr.shape[0], sr.shape[2], _lib.ptr(sr), _lib.ptr(nv),
                                          _lib.ptr(descs)))
        for _ in range(runs):
            ctx.check(ctx.L.bbgpu_eval_run(ctx.h))

    def read(k):
        ss = np.zeros(len(batches[k][3]))
        ctx.check(ctx.L.bbgpu_eval_download(ctx.h, _lib.ptr(ss), None))
        return ss

    alone = []
    for k in range(len(batches)):
        queue(k, 1)
        alone.append(read(k))
    for last in range(len(batches)):
        for k in range(len(batches)):
            queue(k, 20)
        queue(last, 1)
        np.testing.assert_array_equal(read(last), alone[last])
