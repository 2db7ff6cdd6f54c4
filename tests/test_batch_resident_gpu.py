"""Batches on cluster-resident states (the default): against the persistent
kernel, the oracle at the ends of the range, and from a side stream."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from gpu_simulation_b200 import BatchEngine
from gpu_simulation_b200.batch import param_offsets

pytestmark = pytest.mark.gpu

TOL = 1e-10


def circuits(ns, ls, seed):
    rng = np.random.default_rng(seed)
    hs = rng.uniform(-0.5, 2.0, len(ns))
    return hs, rng.uniform(0.0, 2.0 * np.pi, int(param_offsets(ns, ls)[-1]))


@pytest.mark.parametrize("ns,ls", [
    ([n for n in range(2, 17)] * 3, [1 + (5 * k) % 9 for k in range(45)]),
    ([16] * 40, [1 + k % 3 for k in range(40)]),
    ([9] * 700, [1 + k % 5 for k in range(700)]),
    ([13], [64]),
    ([7, 12, 10, 16], [64, 64, 33, 20]),
])
def test_matches_persistent_kernel_and_oracle(ns, ls):
    hs, p = circuits(ns, ls, 17 + len(ns))
    eng = BatchEngine()
    e, g = eng.energy_and_grad(ns, ls, hs, p)
    e2, g2 = eng.energy_and_grad(ns, ls, hs, p)
    assert np.array_equal(e, e2) and np.array_equal(g, g2)
    eng.set_cluster(1)  # an explicit cluster size: the persistent kernel
    e1, g1 = eng.energy_and_grad(ns, ls, hs, p)
    eng.set_resident(True)
    e3, g3 = eng.energy_and_grad(ns, ls, hs, p)
    assert np.array_equal(e, e3) and np.array_equal(g, g3)
    np.testing.assert_allclose(e, e1, atol=TOL, rtol=0)
    np.testing.assert_allclose(g, g1, atol=TOL, rtol=0)
    off = param_offsets(ns, ls)
    for c in range(0, len(ns), max(1, len(ns) // 4)):
        e_ref, g_ref = oracle.energy_and_grad(ns[c], ls[c], hs[c], p[off[c]:off[c + 1]])
        assert abs(e[c] - e_ref) < TOL
        np.testing.assert_allclose(g[off[c]:off[c + 1]], g_ref, atol=TOL, rtol=0)


def test_runs_are_ordered_on_the_callers_stream():
    import torch

    ns, ls = [16, 12, 8, 5] * 8, [3, 4, 5, 6] * 8
    hs, p = circuits(ns, ls, 3)
    eng = BatchEngine()
    e_ref, g_ref = eng.energy_and_grad(ns, ls, hs, p)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        d = torch.zeros(p.size, dtype=torch.float64, device="cuda")
        e = torch.empty(len(ns), dtype=torch.float64, device="cuda")
        g = torch.empty_like(d)
        eng.run_device(d, e, g)  # on zero angles; the next run must not overtake the copy
        d.copy_(torch.from_numpy(p).pin_memory(), non_blocking=True)
        eng.run_device(d, e, g)
        e_out, g_out = e.clone(), g.clone()
    s.synchronize()
    assert np.array_equal(e_out.cpu().numpy(), e_ref) and np.array_equal(g_out.cpu().numpy(), g_ref)
