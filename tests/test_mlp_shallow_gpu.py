"""Products of small depth over many rows (a tile a group of threads)."""

from __future__ import annotations

import pytest

from gpu_simulation_b200.warmstart import WarmStartMLP

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def network(widths, seed):
    import torch

    net = WarmStartMLP(widths)
    g = torch.Generator(device="cuda").manual_seed(seed)
    net.weights.copy_(torch.randn(net.weights.numel(), device="cuda", generator=g))
    return net, g


# 1024 tiles of 32 x 32 and some, or a few less (the other form); depths at the ends of the
# 16-deep stages and of the rule; widths that allow 16-byte stores and that do not
@pytest.mark.parametrize("depth,width,rows", [
    (1, 32, 32768), (3, 64, 16385), (4, 33, 16389), (5, 256, 4097), (16, 31, 32799), (17, 36, 16400), (64, 256, 4096),
    (127, 65, 11000), (128, 64, 16400), (3, 1, 40000), (2, 64, 16352), (100, 130, 6600),
])
def test_shallow_products_match_64_bits(depth, width, rows):
    import torch

    # as the last layer
    net, g = network((depth, width), depth)
    x = torch.randn(rows, depth, device="cuda", generator=g)
    w, b = net.weights[:-width].view(width, depth).double(), net.weights[-width:].double()
    exact = x.double() @ w.T + b
    # at most depth + 1 rounded operations on partial sums of this size
    bound = (depth + 2) * U * (x.double().abs() @ w.abs().T + b.abs())
    out = net.forward(x)
    assert bool(((out.double() - exact).abs() <= bound).all())
    assert torch.equal(net.forward(x), out)
    # as a hidden layer: the sum itself and its GELU
    net, g = network((depth, width, 2), depth + 1)
    w, b = net.weights[:width * depth].view(width, depth).double(), net.weights[width * depth:width * (depth + 1)].double()
    exact = x.double() @ w.T + b
    bound = (depth + 2) * U * (x.double().abs() @ w.abs().T + b.abs())
    work = torch.full((2 * rows * width + 8,), float("nan"), device="cuda")
    net.forward(x, work)
    z, a = work[:rows * width].view(rows, width).double(), work[rows * width:2 * rows * width].view(rows, width).double()
    assert bool(((z - exact).abs() <= bound).all())
    # GELU's slope is at most 1.13; erff is good to 2 units in the last place of a value up to 1
    assert bool(((a - torch.nn.functional.gelu(exact)).abs() <= 1.13 * bound + 8 * U * exact.abs()).all())
    assert bool(torch.isnan(work[2 * rows * width:]).all())  # nothing behind the last row


def test_a_depth_of_three_keeps_up_with_memory():
    """134 MB of outputs: 134 us at 1 TB/s, a sixth of what the device writes."""
    import torch

    net, g = network((3, 256), 9)
    x = torch.randn(131072, 3, device="cuda", generator=g)
    times = []
    for _ in range(5):
        net.forward(x)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            net.forward(x)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) / 10)
    assert min(times) < 0.134, times
