"""Batches on a device that is almost full."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import BatchEngine
from gpu_simulation_b200.batch import param_offsets

pytestmark = pytest.mark.gpu


def fill_device(leave: int):
    """All of the device's free memory but `leave` bytes."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def circuits(ns, ls, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.2, 2.0, len(ns)), rng.uniform(0.0, 2.0 * np.pi, int(param_offsets(ns, ls)[-1]))


def test_one_list_without_room_does_not_change_the_next_ones():
    import torch

    ns, ls = [16] * 160, [1, 2, 3, 4, 5] * 32  # 4 vectors of 1 MiB for each circuit in flight: 144 MiB on clusters of 4
    hs, p = circuits(ns, ls, 1)
    small = ([13, 12, 9, 6], [5, 4, 3, 7])
    hs_small, p_small = circuits(*small, 2)
    fresh = BatchEngine()
    e_ref, g_ref = fresh.energy_and_grad(ns, ls, hs, p)
    e_small, g_small = fresh.energy_and_grad(*small, hs_small, p_small)
    fresh.set_cluster(8)
    e_pers, g_pers = fresh.energy_and_grad(*small, hs_small, p_small)
    assert not np.array_equal(g_small, g_pers)  # the two kernels are told apart by their last bits
    fresh.close()
    eng = BatchEngine()
    full = fill_device(32 << 20)
    e, g = eng.energy_and_grad(ns, ls, hs, p)
    del full
    torch.cuda.empty_cache()
    np.testing.assert_allclose(e, e_ref, atol=1e-10, rtol=0)
    np.testing.assert_allclose(g, g_ref, atol=1e-10, rtol=0)
    assert not np.array_equal(g, g_ref)  # it did take the other kernel
    e, g = eng.energy_and_grad(*small, hs_small, p_small)
    assert np.array_equal(e, e_small) and np.array_equal(g, g_small)
    e, g = eng.energy_and_grad(ns, ls, hs, p)
    assert np.array_equal(e, e_ref) and np.array_equal(g, g_ref)
    eng.close()


def test_a_refused_allocation_is_not_left_for_others_to_find():
    import torch

    eng = BatchEngine()
    many = 4_000_000  # descriptors of 32 and about 40 bytes, allocated half as large again
    full = fill_device(256 << 20)
    with pytest.raises((MemoryError, RuntimeError)):
        eng.set_circuits(np.full(many, 2), np.ones(many), np.ones(many))
    assert int(full[:4].fill_(3).sum()) == 12  # torch checks the last error at its launches
    del full
    torch.cuda.empty_cache()
    eng.close()


def test_a_description_that_failed_is_not_run():
    import torch

    ns, ls = [12, 9], [3, 4]
    hs, p = circuits(ns, ls, 3)
    eng = BatchEngine()
    e_ref, g_ref = eng.energy_and_grad(ns, ls, hs, p)
    d = torch.tensor(p, device="cuda")
    e, g = torch.zeros(2, dtype=torch.float64, device="cuda"), torch.zeros_like(d)
    many = 4_000_000
    full = fill_device(256 << 20)
    with pytest.raises((MemoryError, RuntimeError)):
        eng.set_circuits(np.full(many, 2), np.ones(many), np.ones(many))
    with pytest.raises(ValueError):
        eng.run_device(d, e, g)
    with pytest.raises(ValueError):
        eng.set_cluster(1)
    with pytest.raises(ValueError):
        eng.set_resident(True)
    del full
    torch.cuda.empty_cache()
    assert not g.any()
    e2, g2 = eng.energy_and_grad(ns, ls, hs, p)
    assert np.array_equal(e2, e_ref) and np.array_equal(g2, g_ref)
    with pytest.raises(ValueError):  # refused before anything is touched: the list before stands
        eng.set_circuits([12, 17], [1, 1], [1.0, 1.0])
    eng.run_device(d, e, g)
    assert np.array_equal(g.cpu().numpy(), g_ref)
    eng.close()


def test_reported_bytes_hold_the_resident_circuits_vectors():
    eng = BatchEngine()
    before = eng.device_bytes()
    eng.set_circuits([12] * 4, [2] * 4, [1.0] * 4)
    in_registers = eng.device_bytes()
    eng.set_circuits([16] * 4, [2] * 4, [1.0] * 4)
    tiled = eng.device_bytes()
    eng.close()
    assert before < in_registers < before + (1 << 16)  # descriptors alone
    assert tiled >= in_registers + 4 * (4 << 20)  # psi and lambda, two of each, of 2^16 amplitudes
