"""How the ring contraction's gradient is split over a device's SMs: wire 0's
gradient needs a warp for every column, on the smallest device too."""

from __future__ import annotations

import subprocess

from gpu_simulation_b200.build import CSRC, CUDA_HOME

PROGRAM = r"""
#include "rsv_ring.h"
#include <cstdio>
int main() {
  for (int L = 1; L <= rsv::kRingMaxLayers; ++L)
    for (int n = 12; n <= 31; ++n)
      for (int sms = 1; sms <= 160; ++sms) std::printf("%d %d %d %d\n", L, n, sms, rsv::ring_gradient_ctas(n, L, sms));
}
"""


def test_every_column_of_wire_0_has_a_warp(tmp_path):
    src, exe = tmp_path / "split.cpp", tmp_path / "split"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{CUDA_HOME / 'include'}", str(src), "-o", str(exe)], check=True)
    rows = [tuple(map(int, line.split())) for line in subprocess.run([str(exe)], check=True, capture_output=True,
                                                                     text=True).stdout.splitlines()]
    assert len(rows) == 5 * 20 * 160
    for layers, n, sms, ctas in rows:
        assert 1 <= ctas <= 8
        assert 10 * ctas >= 2 ** (layers - 1), (layers, n, sms)
        if ctas * n > sms:  # more than one round of CTAs only where wire 0 needs it
            assert ctas == (2 if layers == 5 else 1)
