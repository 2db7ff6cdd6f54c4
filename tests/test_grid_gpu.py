"""Circuits of 17 to 20 qubits in one launch over the whole device."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from gpu_simulation_b200 import Engine, ring_ising_energy

pytestmark = pytest.mark.gpu

# At most 64 layers x 20 wires x 3 rounded operations on vectors of norm 1, sums
# of at most 20 terms of size 1: 20 * 3840 * 1.1e-16 = 8.5e-12.
TOL = 1e-10


@pytest.mark.parametrize("n,layers", [(17, 5), (17, 6), (17, 45), (18, 6), (18, 7), (19, 5), (19, 9), (20, 6), (20, 7), (20, 18),
                                      (20, 30), (20, 64)])
def test_matches_passes(n, layers):
    import torch

    p = np.random.default_rng(n + layers).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    p[::7] = 0.0
    p[3::11] = np.pi  # cos of the half angle is 0
    eng = Engine(n, layers, 0.7)
    assert ("tiled" in eng.describe()) == (layers < 64)  # the tables of 64 layers do not fit
    e, g = eng.energy_and_grad(p)
    e2, g2 = eng.energy_and_grad(p)
    assert e == e2 and np.array_equal(g, g2)
    passes = Engine(n, layers, 0.7)
    passes.set_backward_mode("uncompute")
    assert "tiled" not in passes.describe()
    e1, g1 = passes.energy_and_grad(p)
    assert abs(e - e1) < TOL and abs(eng.energy(p) - e1) < TOL
    np.testing.assert_allclose(g, g1, atol=TOL, rtol=0)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    v = ring_ising_energy(x, eng)  # forward and backward in two launches
    x.data.zero_()
    v.backward()
    np.testing.assert_allclose(x.grad.cpu().numpy(), g1, atol=TOL, rtol=0)
    if (n, layers) == (17, 6):
        e_ref, g_ref = oracle.energy_and_grad(n, layers, 0.7, p)
        assert abs(e - e_ref) < TOL
        np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)


def test_in_a_graph_and_on_two_streams():
    import torch

    rng = np.random.default_rng(5)
    engines = [Engine(18, 6, 1.1), Engine(20, 6, 0.4)]
    inputs = [torch.tensor(rng.uniform(0.0, 6.0, 2 * e.num_qubits * 6), device="cuda") for e in engines]
    outs = [(torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(p)) for p in inputs]
    expect = []
    for e, p, (v, g) in zip(engines, inputs, outs):
        e.energy_and_grad_device(p, v, g)
        expect.append((v.item(), g.cpu().numpy()))
    streams = [torch.cuda.Stream() for _ in engines]
    torch.cuda.synchronize()
    for _ in range(10):
        for e, p, (v, g), s in zip(engines, inputs, outs, streams):
            with torch.cuda.stream(s):
                e.energy_and_grad_device(p, v, g)
    torch.cuda.synchronize()
    for (v, g), (ve, ge) in zip(outs, expect):
        assert v.item() == ve and np.array_equal(g.cpu().numpy(), ge)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        engines[0].energy_and_grad_device(inputs[0], *outs[0])
    outs[0][0].zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert outs[0][0].item() == expect[0][0] and np.array_equal(outs[0][1].cpu().numpy(), expect[0][1])
