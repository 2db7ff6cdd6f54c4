"""The tile passes as such: plans that circuits of few layers no longer take by
default (they are contracted along the ring) and that deeper ones from 21 qubits
on do, through explicit schedules, against plain torch in complex128, against
the ring and against the other kernels."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from gpu_simulation_b200 import Engine, ring_ising_energy
from perf.cases import angles, exact

pytestmark = pytest.mark.gpu

TOL = 1e-10


def on_passes(eng):
    return "the plan below is not used" not in eng.describe().splitlines()[0]


def parameters(n, layers, seed=5):
    return angles(2 * n * layers, seed).cpu().numpy()


def reference(n, layers, h, seed=5):
    """Energy and gradient by plain torch in 64 bits; where the ring takes the
    circuit, by that (checked against the oracle elsewhere)."""
    if n <= 26:
        r = exact({"kind": "circuit", "entry": "device", "n": n, "layers": layers, "field": h}, seed)
        return float(r["energy"]), r["grad"].cpu().numpy()
    ring = Engine(n, layers, h)
    assert "ring_contraction" in ring.describe().splitlines()[0]
    e, g = ring.energy_and_grad(parameters(n, layers, seed))
    ring.close()
    return e, g


@pytest.mark.parametrize("n,layers,h", [(23, 4, 0.9), (24, 4, 1.0), (25, 7, 1.3), (26, 5, 0.7), (26, 6, 0.7), (27, 4, 1.0),
                                        (28, 4, 1.1), (29, 4, 0.8)])
def test_tensor_copy_passes(n, layers, h):
    p = parameters(n, layers)
    e_ref, g_ref = reference(n, layers, h)
    eng = Engine(n, layers, h)
    eng.set_backward_mode("checkpoint")
    assert on_passes(eng)
    assert eng.kernels()["tma_passes"] > 0
    results = []
    for tma, fused in ((True, True), (True, False), (False, False)):
        eng.set_kernels(tma=tma, fused_energy=fused)
        assert on_passes(eng) and (eng.kernels()["tma_passes"] > 0) == tma
        e, g = eng.energy_and_grad(p)
        e2, g2 = eng.energy_and_grad(p)
        assert e == e2 and np.array_equal(g, g2)
        assert abs(e - e_ref) < TOL
        np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)
        results.append((e, g))
    for e, g in results[1:]:
        assert abs(e - results[0][0]) < 1e-12
        np.testing.assert_allclose(g, results[0][1], atol=1e-12, rtol=0)
    eng.close()


@pytest.mark.parametrize("n,layers", [(23, 4), (24, 4), (28, 4)])
def test_field_terms_in_the_passes(n, layers):
    """The fused field terms, at n = 28 those of the middle pass too, the energy
    alone, the split forward and backward, and a field changed after planning."""
    import torch

    p = parameters(n, layers)
    eng = Engine(n, layers, 0.8)
    eng.set_backward_mode("checkpoint")
    assert on_passes(eng)
    first = eng.describe().splitlines()[0]
    assert "fused_energy: backward pass 0 applies" in first and (n < 28 or "backward pass 1 applies 7" in first)
    for h in (0.8, 0.55):
        eng.set_field(h)
        e_ref, g_ref = reference(n, layers, h)
        e, g = eng.energy_and_grad(p)
        assert abs(e - e_ref) < TOL and abs(eng.energy(p) - e_ref) < TOL
        np.testing.assert_allclose(g, g_ref, atol=TOL, rtol=0)
        x = torch.tensor(p, device="cuda", requires_grad=True)
        v = ring_ising_energy(x, eng)
        v.backward()
        assert abs(v.item() - e_ref) < TOL
        np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=TOL, rtol=0)
    eng.close()


@pytest.mark.parametrize("n,layers", [(21, 6), (22, 6), (24, 6), (25, 6)])
def test_deeper_circuits_split_forward_and_backward(n, layers):
    """The default path of six layers and more from 21 qubits on."""
    import torch

    p = parameters(n, layers)
    e_ref, g_ref = reference(n, layers, 1.2)
    eng = Engine(n, layers, 1.2)
    assert on_passes(eng)
    e, g = eng.energy_and_grad(p)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    v = ring_ising_energy(x, eng)
    v.backward()
    for energy, grad in ((e, g), (v.item(), x.grad.cpu().numpy())):
        assert abs(energy - e_ref) < TOL
        np.testing.assert_allclose(grad, g_ref, atol=TOL, rtol=0)
    assert abs(eng.energy(p) - e_ref) < TOL
    eng.close()


def test_the_reference_is_the_oracles():
    n, layers, h = 9, 3, 0.7
    e_ref, g_ref = oracle.energy_and_grad(n, layers, h, parameters(n, layers))
    e, g = reference(n, layers, h)
    assert abs(e - e_ref) < 1e-12
    np.testing.assert_allclose(g, g_ref, atol=1e-12, rtol=0)
