"""The refinement's two routes (gather table, plain gathers) give the same
bits, for candidate counts below, at and above the group of 9, and with
per-pattern source points."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("radius,axial", [(1, 1), (1, 2), (1, 3), (2, 3)])
@pytest.mark.parametrize("offsets", [False, True])
def test_routes_agree(radius, axial, offsets):
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200._capi import call, ptr
    from ebsdtorch_b200.ebsd import get_local_orientation_grid

    rng = np.random.default_rng(radius * 10 + axial)
    h, w, n_pix, n, iters = 31, 62, 777, 5, 2
    mp = torch.from_numpy(rng.random((h, w))).float().to(DEV)
    rays = rng.standard_normal((3, n_pix))
    rays = torch.from_numpy(rays / np.linalg.norm(rays, axis=0)).float().to(DEV)
    q = rng.standard_normal((n, 4))
    q = torch.from_numpy(q / np.linalg.norm(q, axis=1, keepdims=True)).float().to(DEV)
    rows = torch.from_numpy(rng.standard_normal((n, n_pix))).float().to(DEV)
    off = torch.from_numpy(0.01 * rng.standard_normal((n, 2))).float().to(DEV) if offsets else None
    grid = get_local_orientation_grid(2.0, radius, axial).float().contiguous().to(DEV)
    got = []
    for name, img in (("ebsd_refine_grid", mp), ("ebsd_refine_grid_quads", kernels.sampling_quads(mp))):
        qo, d = torch.empty_like(q), torch.empty((n, iters), device=DEV)
        call(name, ptr(img), h, w, ptr(rays), n_pix, ptr(off), ptr(rows), rows.stride(0), ptr(q), n, ptr(grid),
             grid.shape[0], 11, 1, iters, 0.5, ptr(qo), ptr(d), None)
        got.append((qo, d))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
