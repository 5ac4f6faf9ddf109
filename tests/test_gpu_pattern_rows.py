"""Detector counts are converted to FP32 rows while they are summed: the same
results as converting first, at row lengths and offsets with and without whole
groups of four, and at one and many row splits."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.uint16, torch.uint8, torch.float16])
@pytest.mark.parametrize("n,side", [(1, 2), (33, 15), (700, 16), (300, 61), (260, 60)])
@pytest.mark.parametrize("skip", [0, 1])
def test_equals_conversion_first(dtype, n, side, skip):
    from ebsdtorch_b200.preprocessing import standard_clean, subtract_overall_background

    g = torch.Generator(DEV).manual_seed(n + side)
    x = torch.rand((n + skip, side, side), device=DEV, generator=g)
    x = x.half() if dtype == torch.float16 else (x * 255).to(torch.int32).to(dtype)
    x = x[skip:]
    # the sums are exact in FP64, so equal whatever their order
    assert torch.equal(subtract_overall_background(x), subtract_overall_background(x.float()))
    if side > 4:
        assert torch.equal(standard_clean(x), standard_clean(x.float()))
