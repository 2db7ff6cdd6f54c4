"""A batch is described anew while a run of it is still in flight: the run keeps
the circuits that it was started with."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import BatchEngine
from gpu_simulation_b200.batch import param_offsets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [0, 148])  # a launch a qubit count; the persistent kernel
@pytest.mark.parametrize("captured", [False, True])
def test_a_run_in_flight_keeps_its_circuits(slots, captured):
    import torch

    rng = np.random.default_rng(11)
    shallow = ([16, 14, 10, 7] * 100, [2, 3, 1, 2] * 100)
    deep = ([7, 16, 13] * 60, [40, 24, 31] * 60)
    lists = []
    eng = BatchEngine(slots=slots)
    for ns, ls in (shallow, deep):
        hs = rng.uniform(0.2, 2.0, len(ns))
        p = rng.uniform(0.0, 2.0 * np.pi, int(param_offsets(ns, ls)[-1]))
        e, g = eng.energy_and_grad(ns, ls, hs, p)
        lists.append((ns, ls, hs, torch.tensor(p, device="cuda"), e, g))
    s = torch.cuda.Stream()
    for i in range(6):  # in turn, no synchronisation between a run and the next description
        ns, ls, hs, p, e_ref, g_ref = lists[i % 2]
        e, g = torch.empty(len(ns), dtype=torch.float64, device="cuda"), torch.empty_like(p)
        eng.set_circuits(ns, ls, hs)
        if captured:
            graph = eng.capture_graph(p, e, g)
            e.zero_()
            with torch.cuda.stream(s):
                s.wait_stream(torch.cuda.default_stream())
                graph.replay()
                graph.replay()
        else:
            s.wait_stream(torch.cuda.current_stream())
            eng.run_device(p, e, g, stream=s)
            eng.run_device(p, e, g, stream=s)
        other = lists[(i + 1) % 2]
        eng.set_circuits(*other[:3])
        torch.cuda.synchronize()
        np.testing.assert_array_equal(e.cpu().numpy(), e_ref)
        np.testing.assert_array_equal(g.cpu().numpy(), g_ref)
        if captured:
            del graph
    eng.close()


@pytest.mark.parametrize("change", ["cluster", "resident"])
def test_another_kernel_is_chosen_with_a_run_in_flight(change):
    import torch

    rng = np.random.default_rng(12)
    ns, ls = [16, 13, 9] * 60, [6, 9, 12] * 60
    hs, p = rng.uniform(0.2, 2.0, len(ns)), rng.uniform(0.0, 6.0, int(param_offsets(ns, ls)[-1]))
    eng = BatchEngine()
    d = torch.tensor(p, device="cuda")
    e, g = torch.empty(len(ns), dtype=torch.float64, device="cuda"), torch.empty_like(d)
    e_ref, g_ref = eng.energy_and_grad(ns, ls, hs, p)
    if change == "resident":
        eng.set_cluster(4)
        e_ref, g_ref = eng.energy_and_grad(ns, ls, hs, p)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    eng.run_device(d, e, g, stream=s)
    if change == "cluster":
        eng.set_cluster(2)
    else:
        eng.set_resident(True)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(e.cpu().numpy(), e_ref)
    np.testing.assert_array_equal(g.cpu().numpy(), g_ref)
    eng.close()
