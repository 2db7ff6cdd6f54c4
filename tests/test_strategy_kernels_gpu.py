"""Each gradient strategy runs its own kernels: an engine of the gate-level walk
or the dense product tree is never moved to the structured strategy's direct
paths, whatever its size, and its forward/backward pair still gives the gradient."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from gpu_simulation_b200 import Engine, ring_ising_energy

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("strategy,name,n,layers", [
    ("inverse_walk_cuQuantum", "gate_level", 2, 1), ("inverse_walk_cuQuantum", "gate_level", 9, 3),
    ("inverse_walk_cuquantum", "gate_level", 13, 2), ("inverse_walk_cuQuantum", "gate_level", 16, 6),
    ("inverse_walk_cuQuantum", "gate_level", 18, 6),
    ("dense_scan", "dense_scan", 2, 1), ("dense_scan", "dense_scan", 5, 4), ("dense_scan", "dense_scan", 8, 3),
])
def test_strategy_keeps_its_kernels(strategy, name, n, layers):
    import torch

    h = 0.8
    p = np.random.default_rng(40 + n).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    e_ref, g_ref = oracle.energy_and_grad(n, layers, h, p)
    eng = Engine(n, layers, h, gradient_strategy=strategy)
    first = eng.describe().splitlines()[0]
    assert name in first and not any(w in first for w in ("ring_contraction", "cluster_resident", "whole_device")), first
    e, g = eng.energy_and_grad(p)
    assert abs(e - e_ref) < TOL and abs(eng.energy(p) - e_ref) < TOL
    np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)
    # forward and backward as a pair, twice, with another call in between
    x = torch.tensor(p, device="cuda", requires_grad=True)
    for interrupted in (False, True):
        x.grad = None
        v = ring_ising_energy(x, eng)
        if interrupted:
            torch.cuda.synchronize()  # the host call runs on the engine's own stream
            eng.energy(p[::-1].copy())
        v.backward()
        assert abs(v.item() - e_ref) < TOL
        np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=TOL, rtol=0)
    # the same kernels after a re-plan
    eng.set_backward_mode("auto")
    assert eng.describe().splitlines()[0] == first
    e2, g2 = eng.energy_and_grad(p)
    assert e2 == e and np.array_equal(g2, g)
    assert eng.benchmark_forward_graph(p, repeats=2)["normal_forward_ms"] > 0.0
    eng.close()
