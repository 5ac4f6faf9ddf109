"""The refinement of up to one pattern an SM and of more run two shapes of one
kernel: the same results for the same patterns, for candidate counts at and
around both group sizes (9 and 16)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n_grid", [1, 3, 9, 11, 15, 17, 27, 125])
@pytest.mark.parametrize("quads", [False, True])
def test_both_shapes_agree(n_grid, quads):
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200._capi import call, ptr

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator().manual_seed(n_grid)
    h, w, n_pix, n, iters = 31, 62, 333, sms + 1, 2
    mp = torch.rand((h, w), generator=g).to(DEV)
    rays = torch.nn.functional.normalize(torch.randn((3, n_pix), generator=g), dim=0).to(DEV)
    q = torch.nn.functional.normalize(torch.randn((n, 4), generator=g), dim=1).to(DEV)
    rows = torch.randn((n, n_pix), generator=g).to(DEV)
    grid = (0.02 * torch.rand((n_grid, 3), generator=g) - 0.01).to(DEV)
    img = kernels.sampling_quads(mp) if quads else mp

    def run(count):
        qo, d = torch.empty((count, 4), device=DEV), torch.empty((count, iters), device=DEV)
        call("ebsd_refine_grid_quads" if quads else "ebsd_refine_grid", ptr(img), h, w, ptr(rays), n_pix, None,
             ptr(rows), n_pix, ptr(q), count, ptr(grid), n_grid, 11, 1, iters, 0.5, ptr(qo), ptr(d), None)
        return qo, d

    (qa, da), (qb, db) = run(sms), run(n)
    assert torch.equal(qa, qb[:sms]) and torch.equal(da, db[:sms])
