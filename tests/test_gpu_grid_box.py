"""The grid generator only visits the cube that can hold the fundamental
zone: the same points, order and cells as the whole grid for every Laue group,
at the smallest edges, odd and even ones, and on both sides of the block-size
switch (2^20 points of the box)."""

import numpy as np
import pytest
import torch

from oracle import di_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("laue", range(1, 12))
@pytest.mark.parametrize("edge", [1, 2, 3, 4, 9, 16, 33])
def test_box_holds_the_zone(laue, edge):
    from ebsdtorch_b200 import kernels

    q, q64, cells = kernels.grid_fz(laue, edge, DEV, want_f64=True, want_cells=True)
    full = O.so3_cubochoric_grid(edge)
    keep = np.flatnonzero(O.ori_in_fz_laue(full, laue))
    assert np.array_equal(cells.cpu().numpy(), keep)
    if keep.size:
        assert np.abs(q64.cpu().numpy() - full[keep]).max() < 1e-12
        assert torch.equal(q.cpu(), q64.float().cpu())


@pytest.mark.parametrize("laue,edge", [(11, 250), (11, 251), (2, 101), (2, 102)])
def test_block_sizes_agree(laue, edge):
    from ebsdtorch_b200 import kernels

    q, _, cells = kernels.grid_fz(laue, edge, DEV, want_cells=True)
    c = cells.cpu().numpy().astype(np.int64)
    assert (np.diff(c) > 0).all()
    i = np.stack([c // (edge * edge), (c // edge) % edge, c % edge], 1)
    pick = np.linspace(0, c.size - 1, 2000).astype(np.int64)
    cu = O.CU_HALF_EDGE * (2.0 * i[pick] - edge) / edge
    assert np.abs(q.cpu().numpy()[pick] - O.qu_std(O.cu2qu(cu))).max() < 1e-6
    # the zone's share of all rotations is 1 / (order of the rotation group)
    assert abs(c.size / edge ** 3 * {11: 24, 2: 2}[laue] - 1) < 0.02
