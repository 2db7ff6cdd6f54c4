"""An energy that no gradient follows stores no H psi: against the energy of the
gradient call, at the sizes where one kernel becomes two."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200 import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,layers", [(13, 2), (17, 2), (20, 3), (21, 2), (21, 6), (22, 6), (23, 6)])
def test_energy_alone(n, layers):
    p = np.random.default_rng(n).uniform(0.0, 2.0 * np.pi, 2 * n * layers)
    eng = Engine(n, layers, 0.9)
    if layers < 6:
        eng.set_backward_mode("uncompute")  # the tile passes
    e, g = eng.energy_and_grad(p)
    # sums of 2^n terms of both signs in a few thousand parts: |H| <= n (1 + 0.9), a
    # part's rounding 1.1e-16 sqrt(2^n / 1000) of its size
    assert abs(eng.energy(p) - e) < 1e-12
    e2, g2 = eng.energy_and_grad(p)
    assert e2 == e and np.array_equal(g2, g)
