"""Stream handles without a GPU."""

from __future__ import annotations

import pytest

from gpu_simulation_b200._lib import raw_stream


def test_a_tensor_on_no_cuda_device_has_no_stream():
    import torch

    with pytest.raises(ValueError):
        raw_stream(torch.zeros(1).get_device())
