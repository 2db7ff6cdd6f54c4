"""Shallow circuits contracted along the ring (rsv_ring.cu): the default of the
structured_adjoint strategy for few layers, checked against the oracle at 1e-10
and against the tile passes, which a caller's explicit plan choice selects."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from gpu_simulation_b200 import Engine

pytestmark = pytest.mark.gpu

TOL = 1e-10


def angles(n, L, seed):
    return np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, 2 * n * L)


@pytest.mark.parametrize("n,L,h", [
    (12, 1, 0.7), (12, 2, 1.1), (12, 3, 0.0), (12, 4, 1.9), (13, 4, -0.8), (14, 3, 1.0), (20, 5, 0.9), (17, 4, 2.0),
    (18, 1, 0.3), (19, 4, 1.2), (21, 2, 1.0), (21, 5, 0.5),
])
def test_matches_oracle(n, L, h):
    p = angles(n, L, 40 * n + L)
    e_ref, g_ref = oracle.energy_and_grad(n, L, h, p)
    eng = Engine(n, L, h)
    assert "ring_contraction" in eng.describe().splitlines()[0]
    e, g = eng.energy_and_grad(p)
    assert abs(e - e_ref) < TOL and abs(eng.energy(p) - e_ref) < TOL
    np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)
    e2, g2 = eng.energy_and_grad(p)
    assert e2 == e and np.array_equal(g2, g)
    eng.close()


@pytest.mark.parametrize("n,L", [(20, 1), (22, 3), (24, 4), (25, 5), (31, 4)])
def test_matches_tile_passes(n, L):
    p = angles(n, L, n + L)
    eng = Engine(n, L, 0.9)
    e, g = eng.energy_and_grad(p)
    eng.set_backward_mode("checkpoint")  # an explicit plan choice: the tile passes
    assert "ring_contraction" not in eng.describe().splitlines()[0]
    e1, g1 = eng.energy_and_grad(p)
    eng.set_backward_mode("auto")
    e2, g2 = eng.energy_and_grad(p)
    eng.close()
    assert e2 == e and np.array_equal(g2, g)
    assert abs(e - e1) < TOL
    np.testing.assert_allclose(g, g1, atol=TOL, rtol=0)


@pytest.mark.parametrize("n,L", [(2, 3), (11, 4), (15, 5), (19, 5), (17, 6)])
def test_other_circuits_keep_the_passes(n, L):
    eng = Engine(n, L, 1.0)
    assert "ring_contraction" not in eng.describe().splitlines()[0]
    eng.close()


@pytest.mark.parametrize("n,L", [(12, 4), (20, 5)])
def test_split_forward_backward_and_graph(n, L):
    import torch

    from gpu_simulation_b200 import ring_ising_energy

    p, h = angles(n, L, 5), 0.8
    e_ref, g_ref = oracle.energy_and_grad(n, L, h, p)
    eng = Engine(n, L, h)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    e = ring_ising_energy(x, eng)
    eng.set_field(3.0)  # the gradient belongs to the forward's field
    e.backward()
    assert abs(e.item() - e_ref) < TOL
    np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=TOL, rtol=0)
    eng.set_field(h)
    # captured once, replayed on other angles
    d = torch.zeros_like(x.detach())
    eo, go = torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty_like(d)
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        eng.energy_and_grad_device(d, eo, go)
    d.copy_(x.detach())
    graph.replay()
    torch.cuda.synchronize()
    assert abs(eo.item() - e_ref) < TOL
    np.testing.assert_allclose(go.cpu().numpy(), g_ref, atol=TOL, rtol=0)
    del graph
    eng.close()


def test_a_nan_angle_voids_energy_and_gradient():
    p = angles(12, 3, 1)
    p[2 * (2 * 12 + 1)] = np.nan  # theta of wire 1 in the last layer
    eng = Engine(12, 3, 1.0)
    e, g = eng.energy_and_grad(p)
    assert np.isnan(e) and np.isnan(g).all()
    eng.close()
