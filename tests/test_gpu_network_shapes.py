"""The fused network kernels at the edges of their tiles and the layer-by-layer ones beside them,
against the FP64 oracle with the kernels' BF16 rounding points (the tolerances of
tests/test_gpu_surrogate.py: they cover FP32 sums of up to 300 terms and the BF16 roundings they flip)."""
import numpy as np
import pytest

from bubbleensemble_implicitextension_b200 import surrogate as SG
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,depth,batch", [(8, 1, 1), (33, 2, 5), (64, 3, 592), (255, 2, 593), (256, 4, 1185),
                                               (96, 2, 2369), (257, 2, 70)])
def test_forward_and_gradients_match_oracle(gpu, width, depth, batch):
    import torch
    net = SG.MLP(width=width, depth=depth, max_batch=2400, seed=width)
    rng = np.random.default_rng(batch)
    norm = [np.asarray(a, np.float32) for a in (rng.normal(0, 1, 6), rng.uniform(0.5, 2, 6), rng.normal(0, 1, 2),
                                                rng.uniform(0.5, 2, 2))]
    net.set_normalization(*norm)
    x = rng.normal(0, 1.5, (batch, 6)).astype(np.float32)
    t = rng.normal(0, 1.0, (batch, 2)).astype(np.float32)
    want, _, _ = M.forward(net.parameters(), net.sizes, x, *norm)
    np.testing.assert_allclose(net.predict(x), want, rtol=2e-3, atol=2e-3 * np.abs(want).max())
    loss = net.backward(torch.as_tensor(x, device="cuda"), torch.as_tensor(t, device="cuda"))
    g = net.gradients()
    want_loss, want = M.backward(net.parameters(), net.sizes, x, t, *norm)
    assert abs(loss - want_loss) <= 1e-4 * max(1.0, want_loss)
    k = 0
    for fi, fo in net.sizes:
        for size in (fi * fo, fo):
            a, b = g[k:k + size].astype(np.float64), want[k:k + size]
            assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-9, (fi, fo, size)
            k += size
