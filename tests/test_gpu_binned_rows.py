"""Binned rows at the edges of the thread rule (loads of a row at and above
4,096 and 16,384), masked and not, against float64 pooling."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.uint16, torch.uint8, torch.float16])
@pytest.mark.parametrize("h,w,b", [(2, 2, 2), (64, 64, 2), (66, 64, 2), (63, 66, 3), (128, 128, 4), (130, 128, 2),
                                   (240, 320, 8), (100, 100, 100)])
@pytest.mark.parametrize("masked", [False, True])
def test_binned_rows(dtype, h, w, b, masked):
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200.kernels import RowBuffers

    g = torch.Generator().manual_seed(h + b)
    vals = torch.randint(0, 200, (3, h, w), generator=g)
    P = (h // b) * (w // b)
    index = torch.arange(0, P, 2) if masked else torch.arange(P)
    n = index.numel()
    f32, norm = torch.empty((3, n), device=DEV), torch.empty(3, device=DEV)
    kernels.prep_patterns(vals.to(torch.int32).to(dtype).to(DEV), RowBuffers(f32=f32, norm=norm), b,
                          index.to(DEV, torch.int32) if masked else None, n, True)
    rows = vals.double().view(3, h // b, b, w // b, b).mean((2, 4)).view(3, P)[:, index]
    ref = rows - rows.mean(1, keepdim=True)
    # pooled values (sums of whole numbers below 2^24 are exact) and mean are
    # rounded once, partial sums of the mean once a value, the difference once
    tol = (3 + -(-n // 512)) * 200 * 2.0 ** -24
    assert (f32.cpu().double() - ref).abs().max() <= tol
    assert (norm.cpu().double() - ref.norm(dim=1)).abs().max() <= tol * n ** 0.5 + 1e-6 * float(ref.norm(dim=1).max())
