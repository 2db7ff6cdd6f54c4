"""The squared error on one cluster and on many, and how fast the large ones are."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_simulation_b200._lib import check, load_library

pytestmark = pytest.mark.gpu


def arrays(count, seed, offset=0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(count + offset, device="cuda", generator=g)[offset:] for _ in range(2)]


def mse(out, target, dout, loss, partials):
    import torch

    check(load_library().rsv_mlp_mse(out.numel(), out.data_ptr(), target.data_ptr(), dout.data_ptr(), loss.data_ptr(),
                                     partials.data_ptr(), torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("offset", [0, 1])  # 16-byte loads, or an array that does not allow them
@pytest.mark.parametrize("count", [1, 3, 4097, (3 << 17) - 1, 3 << 17, (7 << 16) - 1, 7 << 16, (7 << 16) + 5,
                                   (36 << 16) - 1, (36 << 16) + 3, 20_000_001])
def test_matches_64_bits(count, offset):
    import torch

    out, target = arrays(count, count % 1000, offset)
    dout, loss, partials = torch.full_like(out, 7.0), torch.zeros(1, device="cuda"), torch.zeros(256, device="cuda")
    mse(out, target, dout, loss, partials)
    diff = out.double() - target.double()
    # a difference, its square and the sums of at most 140 of them in a thread, then over its warp,
    # CTA, cluster and the clusters: fewer than 256 roundings one after the other, all of one sign
    assert abs(loss.item() - diff.square().mean().item()) <= diff.square().mean().item() * 256 * 2.0 ** -24
    # (three roundings)
    np.testing.assert_allclose(dout.cpu().numpy(), (2.0 * diff / count).cpu().numpy(), rtol=4 * 2.0 ** -24, atol=1e-7 / count)
    first = loss.item()
    mse(out, target, dout, loss, partials)
    assert loss.item() == first


def test_large_arrays_reach_more_than_a_cluster_of_sms():
    """Three arrays of 128 MiB.  Eight SMs move at most 8 * 64 bytes a clock, 1 TB/s
    at 1.965 GHz, which takes 400 us; the whole device's 6.5 TB/s take 62 us."""
    import torch

    out, target = arrays(1 << 25, 1)
    dout, loss, partials = torch.empty_like(out), torch.zeros(1, device="cuda"), torch.zeros(256, device="cuda")
    times = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        mse(out, target, dout, loss, partials)
        a.record()
        mse(out, target, dout, loss, partials)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    assert min(times) < 0.25, times
