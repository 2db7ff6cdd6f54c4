"""Engines on the ring and cluster paths hold the memory that those need, not the
tile passes' state buffers, and read none of it before it is written."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import Engine, ring_ising_energy

pytestmark = pytest.mark.gpu

TOL = 1e-10


def free_bytes():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("n,layers", [(5, 7), (8, 8), (12, 3), (12, 8), (14, 6), (15, 6), (16, 4), (16, 6), (18, 6), (20, 5),
                                      (20, 6), (24, 4), (28, 2)])
def test_memory_and_results_on_used_memory(n, layers):
    import torch

    p = np.random.default_rng(n + layers).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    junk = torch.full((1 << 28,), float("nan"), dtype=torch.float64, device="cuda")  # 2 GiB, for the allocations to reuse
    torch.cuda.synchronize()
    del junk
    before = free_bytes()
    eng = Engine(n, layers, 0.7)
    # ring: 2 * 136 * 20 * 5 * 4 KiB at most; cluster: 6 vectors and 6 MiB of records at most
    assert eng.device_bytes() < 128 << 20
    assert before - free_bytes() < 256 << 20
    e, g = eng.energy_and_grad(p)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    v = ring_ising_energy(x, eng)
    v.backward()
    times = eng.benchmark_forward_graph(p, repeats=2)  # the tile passes' forward, on buffers of its own
    assert times["normal_forward_ms"] > 0.0 and times["graph_forward_ms"] > 0.0
    assert eng.device_bytes() < 128 << 20
    e2, g2 = eng.energy_and_grad(p)
    assert e2 == e and np.array_equal(g2, g)
    eng.set_backward_mode("uncompute")
    assert eng.device_bytes() >= 2 * 16 << max(n, 12)
    e1, g1 = eng.energy_and_grad(p)
    eng.set_backward_mode("auto")
    assert eng.device_bytes() < 128 << 20
    e3, g3 = eng.energy_and_grad(p)
    eng.close()
    assert e3 == e and np.array_equal(g3, g)
    assert abs(e - e1) < TOL and abs(v.item() - e1) < TOL
    np.testing.assert_allclose(g, g1, atol=TOL, rtol=0)
    np.testing.assert_allclose(x.grad.cpu().numpy(), g1, atol=TOL, rtol=0)


def test_a_ring_circuit_runs_on_an_almost_full_device():
    import torch

    n, layers = 28, 4
    p = np.random.default_rng(2).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 1.0)
    e_ref, g_ref = eng.energy_and_grad(p)
    eng.close()
    full = torch.empty(free_bytes() - (512 << 20), dtype=torch.uint8, device="cuda")
    eng = Engine(n, layers, 1.0)
    e, g = eng.energy_and_grad(p)
    eng.close()
    del full
    torch.cuda.empty_cache()
    assert e == e_ref and np.array_equal(g, g_ref)


def test_a_schedule_that_does_not_fit_is_refused_and_so_are_calls_until_one_does():
    """28 qubits, 40 layers: the checkpoints (two buffers of 4 GiB a layer) are
    more than any device's memory."""
    import torch

    from gpu_simulation_b200._lib import EngineError, check

    n, layers = 28, 40
    p = np.random.default_rng(4).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 1.0)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    v = ring_ising_energy(x, eng)
    with pytest.raises(EngineError):
        eng.set_backward_mode("checkpoint")
    d, e, g = x.detach(), torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(x.detach())
    for call in (lambda: eng.energy(p), lambda: eng.energy_and_grad(p), lambda: eng.energy_and_grad_device(d, e, g),
                 lambda: eng.profile_energy_and_grad(p), lambda: eng.benchmark_forward_graph(p, repeats=1),
                 lambda: ring_ising_energy(x, eng), v.backward):
        with pytest.raises(EngineError):
            call()
    assert not g.any()
    assert eng.device_bytes() < 1 << 30
    eng.set_backward_mode("auto")
    assert abs(eng.energy(p) - v.item()) < 1e-12
    with pytest.raises(ValueError):
        check(eng._lib.rsv_set_backward_mode(eng._h, 9))
    assert abs(eng.energy(p) - v.item()) < 1e-12  # an unknown mode changes nothing
    eng.close()
