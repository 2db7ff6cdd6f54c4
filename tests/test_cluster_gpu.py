"""Circuits of up to 16 qubits whose state stays in one thread-block cluster
(rsv_cluster.cu): the default of the structured_adjoint strategy for the deeper
small circuits, checked against the oracle at 1e-10."""

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
    (2, 1, 0.7), (2, 7, 1.0), (3, 1, 1.0), (3, 6, 0.4), (6, 2, 0.9), (9, 1, 0.2), (11, 4, 1.0), (4, 9, 1.2), (5, 6, 0.0), (6, 8, -0.7), (7, 6, 1.5), (7, 64, 1.0),
    (8, 8, 1.0), (9, 7, 0.8), (10, 6, 1.1), (11, 9, 2.0), (12, 6, 0.3), (12, 64, 1.0), (13, 6, 0.9), (14, 7, 1.0),
    (15, 5, 1.3), (16, 6, 0.6), (16, 11, 1.0),
])
def test_matches_oracle(n, L, h):
    p = angles(n, L, 50 * n + L)
    e_ref, g_ref = oracle.energy_and_grad(n, L, h, p)
    eng = Engine(n, L, h)
    assert "cluster_resident" in eng.describe().splitlines()[0]
    e, g = eng.energy_and_grad(p)
    assert abs(e - e_ref) < TOL and abs(eng.energy(p) - e_ref) < TOL
    np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)
    e2, g2 = eng.energy_and_grad(p)
    assert e2 == e and np.array_equal(g2, g)
    eng.set_backward_mode("uncompute")  # an explicit plan choice: the tile passes
    e3, g3 = eng.energy_and_grad(p)
    eng.close()
    assert abs(e3 - e) < TOL
    np.testing.assert_allclose(g3, g, atol=TOL, rtol=0)


@pytest.mark.parametrize("n,L", [(17, 6), (12, 65)])
def test_other_circuits_keep_the_passes(n, L):
    eng = Engine(n, L, 1.0)
    assert "cluster_resident" not in eng.describe().splitlines()[0]
    eng.close()


@pytest.mark.parametrize("special", [0.0, np.pi / 2, np.pi, 2 * np.pi, -3 * np.pi])
def test_angles_at_the_ends_of_the_tangent_form(special):
    n, L = 10, 6
    p = np.full(2 * n * L, special)
    p[::3] += 0.25
    e_ref, g_ref = oracle.energy_and_grad(n, L, 1.0, p)
    eng = Engine(n, L, 1.0)
    e, g = eng.energy_and_grad(p)
    eng.close()
    assert abs(e - e_ref) < TOL
    np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)


@pytest.mark.parametrize("n,L", [(5, 7), (12, 6), (15, 6)])
def test_split_forward_backward_and_graph(n, L):
    import torch

    from gpu_simulation_b200 import ring_ising_energy

    p, h = angles(n, L, 5), 0.8
    e_ref, g_ref = oracle.energy_and_grad(n, L, h, p)
    eng = Engine(n, L, h)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    e = ring_ising_energy(x, eng)
    x.data.zero_()  # the gradient belongs to the forward's angles and field
    eng.set_field(3.0)
    e.backward()
    assert abs(e.item() - e_ref) < TOL
    np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=TOL, rtol=0)
    eng.set_field(h)
    d = torch.zeros_like(x.detach())
    eo, go = torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty_like(d)
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        eng.energy_and_grad_device(d, eo, go)
    d.copy_(torch.tensor(p))
    graph.replay()
    torch.cuda.synchronize()
    assert abs(eo.item() - e_ref) < TOL
    np.testing.assert_allclose(go.cpu().numpy(), g_ref, atol=TOL, rtol=0)
    del graph
    eng.close()


def test_a_nan_angle_voids_energy_and_gradient():
    p = angles(11, 6, 1)
    p[7] = np.nan
    eng = Engine(11, 6, 1.0)
    e, g = eng.energy_and_grad(p)
    assert np.isnan(e) and np.isnan(g).all()
    eng.close()
