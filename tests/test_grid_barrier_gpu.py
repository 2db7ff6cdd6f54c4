"""A whole-device call whose blocks do not meet in time: all of its results are
void, the host is told, and the calls after it are as they were.

The patience of a barrier is set to nothing: a block that does not find all
others there gives up.  At 20 qubits, where some blocks have a second tile, the
first one to arrive always does; below, blocks can also meet at once."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import Engine
from gpu_simulation_b200._lib import EngineError, check

pytestmark = pytest.mark.gpu

PATIENCE = 1 << 21


def set_polls(eng, polls):
    check(eng._lib.rsv_set_barrier_polls(eng._h, polls))


@pytest.mark.parametrize("n,layers", [(17, 5), (18, 6), (19, 5), (20, 6)])
def test_a_call_is_void_as_a_whole_or_not_at_all(n, layers):
    import torch

    p = np.random.default_rng(n).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 0.9)
    assert "whole_device" in eng.describe().splitlines()[0]
    d = torch.tensor(p, device="cuda")
    e_ref, g_ref = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(d)
    eng.energy_and_grad_device(d, e_ref, g_ref)
    set_polls(eng, 0)
    for _ in range(50):
        e, g = torch.zeros_like(e_ref), torch.zeros_like(d)
        eng.energy_and_grad_device(d, e, g)
        lost = bool(torch.isnan(e).all())
        if lost:
            assert torch.isnan(g).all()
        else:
            assert torch.equal(e, e_ref) and torch.equal(g, g_ref)
        assert lost or n < 20
    set_polls(eng, PATIENCE)
    eng.energy_and_grad_device(d, e, g)
    assert torch.equal(e, e_ref) and torch.equal(g, g_ref)
    eng.close()


def test_host_calls_are_told_and_later_ones_not_affected():
    import torch

    n, layers = 20, 6
    p = np.random.default_rng(n).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 0.9)
    e_ref, g_ref = eng.energy_and_grad(p)
    set_polls(eng, 0)
    with pytest.raises(EngineError):
        eng.energy_and_grad(p)
    with pytest.raises(EngineError):
        eng.energy(p)
    with pytest.raises(EngineError):
        eng.profile_energy_and_grad(p)
    # nothing of it stays: with the usual patience, and on the tile passes
    set_polls(eng, PATIENCE)
    e2, g2 = eng.energy_and_grad(p)
    assert e2 == e_ref and np.array_equal(g2, g_ref)
    set_polls(eng, 0)
    d = torch.tensor(p, device="cuda")
    eng.energy_and_grad_device(d, torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(d))
    torch.cuda.synchronize()
    eng.set_backward_mode("uncompute")
    e3, g3 = eng.energy_and_grad(p)
    assert abs(e3 - e_ref) < 1e-10
    np.testing.assert_allclose(g3, g_ref, atol=1e-10, rtol=0)
    # a NaN angle is no lost call
    eng.set_backward_mode("auto")
    set_polls(eng, PATIENCE)
    q = p.copy()
    q[3] = np.nan
    e4, g4 = eng.energy_and_grad(q)
    assert np.isnan(e4) and np.isnan(g4).all()
    with pytest.raises(ValueError):
        set_polls(eng, -1)
    eng.close()


def test_a_backward_that_gives_up_keeps_the_forwards_energy():
    import torch

    from gpu_simulation_b200 import ring_ising_energy

    n, layers = 20, 6
    p = np.random.default_rng(3).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 0.9)
    e_ref, g_ref = eng.energy_and_grad(p)
    x = torch.tensor(p, device="cuda", requires_grad=True)
    v = ring_ising_energy(x, eng)
    set_polls(eng, 0)
    v.backward()
    assert abs(v.item() - e_ref) < 1e-12 and torch.isnan(x.grad).all()
    set_polls(eng, PATIENCE)
    x.grad = None
    ring_ising_energy(x, eng).backward()
    np.testing.assert_allclose(x.grad.cpu().numpy(), g_ref, atol=1e-12, rtol=0)
    eng.close()
