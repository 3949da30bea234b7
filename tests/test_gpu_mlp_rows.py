"""The three-kernel step of the surrogate network (``csrc/mlp.cu``: k_rows, k_wgrad, k_adam) at the sizes where its tiles
can go wrong (rows that do not fill a tile or a split of the batch, inputs that do not fill a slice, both widths), against
the float64 network with the kernels' BF16 roundings: the bounds of the gradient test of the layer-by-layer path."""
import numpy as np
import pytest

import test_gpu_mlp as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,d,n", [(256, 8, 1000), (256, 1, 17), (256, 128, 129), (128, 33, 1500), (128, 44, 256),
                                        (256, 42, 2500)])
def test_gradients(gpu_lib, monkeypatch, hidden, d, n):
    from bbarolo2_gb300.surrogate import MLP
    monkeypatch.setattr(ref, "H", hidden)
    monkeypatch.setattr(ref, "D", d)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, d)).astype(np.float32)
    t = np.sin(x[:, 0]).astype(np.float32)
    net = MLP(d, hidden, seed=3)
    p = net.params()
    g, loss = net.gradients(x, t)
    loss_r, g_r, _ = ref._reference(p, x, t, rounded=True)
    assert abs(loss - loss_r) <= 1e-4 * loss_r
    o = 0
    for s in (hidden * d, hidden, hidden * hidden, hidden, hidden * hidden, hidden, hidden, 1):
        np.testing.assert_allclose(g[o:o + s], g_r[o:o + s], rtol=0, atol=5e-3 * np.abs(g_r[o:o + s]).max())
        o += s
