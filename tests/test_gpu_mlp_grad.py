"""The gradient kernel at the batch sizes where its chunks change over: one
sample, parts of a warp, one chunk per CTA that is not full, the last chunk
ragged, several chunks per CTA.  Tolerance: FP32 sums of n products, each
rounded (2^-24), of a gradient whose norm the sums do not cancel by more than a
factor of a hundred: 1e-5 of its norm, as in the test of the 512-sample batch."""
import numpy as np
import pytest

import pymlp
from rapidsolid import configs, surrogate

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 500, 513, 4095, 4096, 4097, 9001])
def test_gradient_at_chunk_edges(n):
    p = configs.scale_fp32()
    box = surrogate.default_box()
    x, y = surrogate.sample(p, box, n, seed=17)
    box.y_mean[0], box.y_mean[1], box.y_scale[0], box.y_scale[1] = 100.0, -50.0, 3000.0, 800.0
    w = surrogate.init_weights(5)
    w += np.random.default_rng(6).normal(0, 0.05, w.shape).astype(np.float32)
    g, loss = surrogate.grad(box, torch.from_numpy(w).cuda(), x, y)
    l_ref, g_ref = pymlp.loss_and_grad(w, x.cpu().numpy(), y.cpu().numpy(), box.y_mean[:], box.y_scale[:])
    assert abs(loss.item() - l_ref) <= 1e-5 * l_ref
    g = g.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)
    for a, b in ((0, 96), (96, 128), (128, 1152), (1152, 1184), (1184, 1248), (1248, 1250)):
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) <= 1e-5 * np.linalg.norm(g_ref), (a, b)
