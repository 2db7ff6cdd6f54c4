"""Angles that are not finite: the circuit's energy and whole gradient are NaN, on
every path; the circuits beside it in a batch, which take over its vectors and
tables, are as without it."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import BatchEngine, Engine
from gpu_simulation_b200.batch import param_offsets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n,layers", [(6, 1), (9, 5), (12, 8), (14, 5), (15, 6), (16, 6), (18, 6), (20, 7), (16, 3), (20, 5), (21, 6)])
def test_one_circuit(n, layers, bad):
    rng = np.random.default_rng(n)
    p = rng.uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 0.9)
    e_ref, g_ref = eng.energy_and_grad(p)
    for at in (0, int(rng.integers(p.size)), p.size - 1):
        q = p.copy()
        q[at] = bad
        e, g = eng.energy_and_grad(q)
        assert np.isnan(e) and np.isnan(g).all(), at
    e, g = eng.energy_and_grad(p)
    assert e == e_ref and np.array_equal(g, g_ref)
    eng.close()


@pytest.mark.parametrize("ns,ls", [([16] * 200, [2] * 200), ([13, 14, 15, 16] * 60, [1, 3, 2, 4] * 60),
                                   ([5, 9, 11, 12, 13] * 80, [3, 2, 6, 4, 5] * 80)])
def test_in_a_batch(ns, ls):
    rng = np.random.default_rng(len(ns))
    off = param_offsets(ns, ls)
    hs, p = rng.uniform(0.2, 2.0, len(ns)), rng.uniform(0.0, 2.0 * np.pi, int(off[-1]))
    eng = BatchEngine()
    e_ref, g_ref = eng.energy_and_grad(ns, ls, hs, p)
    bad = rng.choice(len(ns), len(ns) // 4, replace=False)
    q = p.copy()
    for c in bad:
        q[rng.integers(off[c], off[c + 1])] = rng.choice([np.nan, np.inf])
    e, g = eng.energy_and_grad(ns, ls, hs, q)
    eng.close()
    for c in range(len(ns)):
        part = slice(off[c], off[c + 1])
        if c in bad:
            assert np.isnan(e[c]) and np.isnan(g[part]).all(), c
        else:
            assert e[c] == e_ref[c] and np.array_equal(g[part], g_ref[part]), c
