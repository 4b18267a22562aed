"""The multiplier of the two-level quantiser, float32(1) / float32(tensor_scale), on the host."""
import numpy as np
import pytest
import torch

from gpu_kernels_b200.nvfp4 import inverse_tensor_scale


@pytest.mark.parametrize("value", [1.0, 3.0, 0.0007, 1e-30, 448.0])
def test_any_scalar_gives_the_same_reciprocal(value):
    want = float(np.float32(1.0) / np.float32(value))
    assert inverse_tensor_scale(value) == want
    for scalar in (torch.tensor(value, dtype=torch.float64), torch.tensor([value], dtype=torch.float64),
                   torch.tensor(value, dtype=torch.float64, requires_grad=True), np.float64(value), str(value)):
        assert inverse_tensor_scale(scalar) == want, scalar
    half = torch.tensor(value, dtype=torch.bfloat16)
    assert inverse_tensor_scale(half) == float(np.float32(1.0) / np.float32(float(half)))


def test_scales_the_kernel_refuses():
    # the entry point takes positive finite multipliers: these come out as 0, inf or NaN, without a warning
    assert inverse_tensor_scale(0.0) == float("inf") and inverse_tensor_scale(float("inf")) == 0.0
    assert np.isnan(inverse_tensor_scale(float("nan")))
