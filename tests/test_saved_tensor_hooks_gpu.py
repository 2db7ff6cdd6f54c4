"""The autograd Function under saved-tensor hooks: what they hand back is used
where it is fit to be, and refused where it is not."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import Engine, ring_ising_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,layers", [(6, 3), (12, 3), (16, 6), (18, 6), (21, 6)])
def test_hooks(n, layers):
    import torch

    p = np.random.default_rng(n).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 0.9)
    _, g_ref = eng.energy_and_grad(p)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    with torch.autograd.graph.save_on_cpu():
        v = ring_ising_energy(x, eng)
    v.backward()
    np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=1e-12, rtol=0)
    for unpack in (lambda t: t.cpu(), lambda t: t.float()):
        x.grad = None
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            v = ring_ising_energy(x, eng)
        with pytest.raises(ValueError):
            v.backward()
        assert x.grad is None
    x.grad = None
    ring_ising_energy(x, eng).backward()
    np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=1e-12, rtol=0)
    eng.close()
