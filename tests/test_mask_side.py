"""Cells per side of the occupancy mask: the FP32 product's whole part, for
every number that float() takes, and what is no such number refused."""
import numpy as np
import pytest
import torch

from diver_gb300.ray_voxel_intersection import mask_side


@pytest.mark.parametrize("scale", [1.0, 0.5, 0.25, 1 / 3, 0.1, 0.7, 1e-9])
@pytest.mark.parametrize("n", [1, 3, 10, 64, 255, 256, 257, 1000, 4095])
def test_side_is_the_fp32_product(n, scale):
    assert mask_side(n, scale) == int(np.float32(n) * np.float32(scale))


@pytest.mark.parametrize("n", [64, 64.0, "64", np.float32(64), np.int64(64), torch.tensor(64), torch.tensor([64.0])])
def test_side_of_what_float_takes(n):
    assert mask_side(n, "0.5") == 32


@pytest.mark.parametrize("n,scale", [(float("inf"), 1.0), (1e39, 1.0), (float("nan"), 1.0), ("x", 1.0), (None, 1.0)])
def test_no_side(n, scale):
    with pytest.raises((OverflowError, ValueError, TypeError)):
        mask_side(n, scale)
