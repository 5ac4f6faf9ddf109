"""The sums behind prepared rows: no FP32 partial sum of the mean or the norm
takes more than ceil(n / 512) values of a row, whatever the block size."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _prep(x, subtract, index=None):
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200.kernels import RowBuffers

    n, n_pix = x.shape[0], (x.shape[1] * x.shape[2] if index is None else index.numel())
    f32, norm = torch.empty((n, n_pix), device=DEV), torch.empty(n, device=DEV)
    kernels.prep_patterns(x.to(DEV), RowBuffers(f32=f32, norm=norm), 1, index, n_pix, subtract)
    return f32.cpu(), norm.cpu()


SMALL = 0.99 * 2.0 ** -24  # just below half a unit in the last place of one


@pytest.mark.parametrize("side", [33, 60, 61, 64, 127, 128, 129, 160])
@pytest.mark.parametrize("masked", [False, True])
def test_mean_of_values_that_an_fp32_sum_loses(side, masked):
    """Ones, then values that one plus each of them loses: a partial sum of m
    values is off by at most (m - 1) 2^-24 of itself."""
    n = side * side
    x = torch.full((n,), SMALL)
    threads = 128 if n <= 4096 else 256 if n <= 16384 else 512
    x[:threads] = 1.0
    x[n - 1] = 0.0  # its difference to the mean is the mean
    index = torch.arange(n, dtype=torch.int32, device=DEV) if masked else None
    f32, _ = _prep(x.view(1, side, side), True, index)
    exact = float(x.double().mean())
    longest = -(-n // 512)
    # the last term: the rounding of the mean itself
    assert abs(-float(f32[0, n - 1]) - exact) <= (longest - 1 + 1) * 2.0 ** -24 * exact


def test_infinite_values_spread_as_in_a_plain_mean():
    x = torch.ones((1, 8, 8))
    x[0, 3, 3] = float("inf")
    f32, _ = _prep(x, True)
    assert torch.isnan(f32[0, 27]) and bool((torch.cat([f32[0, :27], f32[0, 28:]]) == -float("inf")).all())


@pytest.mark.parametrize("side", [64, 128, 160])
def test_norm_of_values_that_an_fp32_sum_loses(side):
    """A one, then squares just below half a unit in the last place of one: a
    chain of m values loses all but the first, (m - 1) 2^-24 of its sum."""
    n = side * side
    x = torch.full((n,), float(np.sqrt(SMALL)), dtype=torch.float32)
    threads = 128 if n <= 4096 else 256 if n <= 16384 else 512
    x[:4 * threads:4] = 1.0
    _, norm = _prep(x.view(1, side, side), False)
    exact = float(x.double().square().sum().sqrt())
    longest = -(-n // 512)
    assert abs(float(norm[0]) - exact) <= (0.5 * longest + 1) * 2.0 ** -24 * exact
