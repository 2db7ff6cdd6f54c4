"""Circuits of 13 to 16 qubits whose state passes through a cluster in tiles:
alone and in batches of the sizes that choose each number of CTAs."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from gpu_simulation_b200 import BatchEngine, Engine
from gpu_simulation_b200.batch import param_offsets

pytestmark = pytest.mark.gpu

# At most 64 layers x 16 wires x 3 rounded operations on vectors of norm 1, sums
# of at most 16 terms of size 1: 16 * 3072 * 1.1e-16 = 5e-12.
TOL = 1e-10


def angles(count, seed):
    p = np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, count)
    p[::7] = 0.0
    p[3::11] = np.pi  # cos of the half angle is 0
    return p


@pytest.mark.parametrize("n,layers,count", [
    (13, 3, 400), (13, 64, 2), (13, 2, 200), (14, 2, 160), (14, 3, 70), (14, 21, 37), (15, 2, 160), (15, 20, 80),
    (15, 3, 40), (15, 21, 8), (16, 1, 300), (16, 2, 150), (16, 3, 64), (16, 21, 40), (16, 64, 9), (16, 5, 8), (16, 7, 1),
])
def test_equal_circuits_in_a_batch(n, layers, count):
    ns, ls = [n] * count, [layers] * count
    hs = np.linspace(-0.5, 2.0, count)
    p = angles(2 * n * layers * count, n + layers + count)
    eng = BatchEngine()
    e, g = eng.energy_and_grad(ns, ls, hs, p)
    e2, g2 = eng.energy_and_grad(ns, ls, hs, p)
    assert np.array_equal(e, e2) and np.array_equal(g, g2)
    eng.set_cluster(1)  # the persistent kernel
    e1, g1 = eng.energy_and_grad(ns, ls, hs, p)
    np.testing.assert_allclose(e, e1, atol=TOL, rtol=0)
    np.testing.assert_allclose(g, g1, atol=TOL, rtol=0)
    off = param_offsets(ns, ls)
    if layers <= 21:
        e_ref, g_ref = oracle.energy_and_grad(n, layers, hs[-1], p[off[-2]:])
        assert abs(e[-1] - e_ref) < TOL
        np.testing.assert_allclose(g[off[-2]:], g_ref, atol=TOL, rtol=0)


@pytest.mark.parametrize("layers", [5, 6, 7, 20, 64])
def test_one_circuit_of_16_qubits(layers):
    import torch

    from gpu_simulation_b200 import ring_ising_energy

    n, h = 16, 0.7
    p = angles(2 * n * layers, layers)
    eng = Engine(n, layers, h)
    assert "tiled" in eng.describe()
    e, g = eng.energy_and_grad(p)
    passes = Engine(n, layers, h)
    passes.set_backward_mode("uncompute")
    assert "tiled" not in passes.describe()
    e1, g1 = passes.energy_and_grad(p)
    assert abs(e - e1) < TOL
    np.testing.assert_allclose(g, g1, atol=TOL, rtol=0)
    assert abs(eng.energy(p) - e) < TOL  # without the backward
    x = torch.tensor(p, dtype=torch.float64, device="cuda", requires_grad=True)
    v = ring_ising_energy(x, eng)  # forward and backward in two launches
    x.data.zero_()
    v.backward()
    np.testing.assert_allclose(x.grad.cpu().numpy(), g, atol=TOL, rtol=0)
