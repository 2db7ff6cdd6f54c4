"""The network's products where a cluster of 2, 4 or 8 CTAs shares the depth: at
the depths where each begins, with ragged tiles, against the float64 oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,batch", [
    ((3, 127, 5), 127), ((3, 128, 5), 128), ((3, 129, 33), 255), ((5, 256, 40), 256), ((3, 40, 7), 511),
    ((3, 40, 7), 512), ((7, 513, 33), 700), ((3, 256, 256, 192), 513), ((200, 300, 100), 1100),
])
def test_loss_and_gradient_match_oracle(widths, batch):
    import torch

    from gpu_simulation_b200.warmstart import WarmStartMLP

    net = WarmStartMLP(widths, seed=5)
    rng = np.random.default_rng(6)
    x = rng.uniform(-1.0, 2.0, (batch, widths[0])).astype(np.float32)
    t = rng.uniform(-3.0, 3.0, (batch, widths[-1])).astype(np.float32)
    loss, grad = net.gradient(torch.from_numpy(x), torch.from_numpy(t))
    again = net.gradient(torch.from_numpy(x), torch.from_numpy(t))[1]
    assert torch.equal(grad, again)
    w64 = net.weights.cpu().numpy().astype(np.float64)
    out, cache = mlp.forward(w64, widths, x.astype(np.float64))
    l_ref, dout = mlp.mse(out, t.astype(np.float64))
    g_ref = mlp.backward(w64, widths, cache, dout)
    # float32 sums of at most 1100 terms: sqrt(1100) * 6e-8 of the largest entry, with room
    assert abs(loss.item() - l_ref) < 1e-5 * abs(l_ref)
    np.testing.assert_allclose(grad.cpu().numpy(), g_ref, atol=1e-5 * np.abs(g_ref).max(), rtol=1e-3)
