"""The NLPAR window passes at the edges of their tiles: every radius, scans
smaller than a tile and not multiples of one, pattern lengths off the chunk
and off the 16-byte accesses, blocks of offsets, repeated offsets and offsets
outside the window, against float64 sums."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _shift(g, di, dj):
    hs, ws = g.shape[:2]
    s = torch.zeros_like(g)
    y0, y1, x0, x1 = max(0, -di), min(hs, hs - di), max(0, -dj), min(ws, ws - dj)
    if y0 < y1 and x0 < x1:
        s[y0:y1, x0:x1] = g[y0 + di:y1 + di, x0 + dj:x1 + dj]
    return s


@pytest.mark.parametrize("r", range(0, 8))
@pytest.mark.parametrize("hs,ws,n_pix,ld_extra", [(1, 1, 4, 0), (3, 1, 64, 0), (7, 9, 63, 0), (13, 17, 68, 4),
                                                  (9, 33, 130, 1), (25, 10, 129, 0)])
def test_window_passes(r, hs, ws, n_pix, ld_extra):
    from ebsdtorch_b200._capi import call, ptr

    g = torch.Generator().manual_seed(r * 100 + hs)
    x = torch.rand((hs * ws, n_pix + ld_extra), generator=g).to(DEV)
    off = torch.stack(torch.meshgrid(torch.arange(-r, r + 1), torch.arange(-r, r + 1), indexing="ij"), -1)
    off = off.reshape(-1, 2)[torch.randperm((2 * r + 1) ** 2, generator=g)]
    K = off.shape[0]
    od = off.to(device=DEV, dtype=torch.int32).contiguous()
    w = torch.softmax(torch.rand((hs * ws, K), generator=g), 1).to(DEV)
    d = torch.full((hs * ws, K), -1.0, device=DEV)
    out = torch.full((hs * ws, n_pix), -1.0, device=DEV)
    call("ebsd_nlpar_dists_window", ptr(x), hs, ws, n_pix, x.stride(0), r, ptr(od), K, ptr(d), None)
    call("ebsd_nlpar_average_window", ptr(x), hs, ws, n_pix, x.stride(0), r, ptr(od), K, ptr(w), ptr(out), n_pix, None)
    # the same in blocks of offsets
    d2, out2 = torch.full_like(d, -1.0), torch.full_like(out, -1.0)
    step = max(1, min(128, K // 2))
    for o0 in range(0, K, step):
        n = min(step, K - o0)
        call("ebsd_nlpar_dists", ptr(x), hs, ws, n_pix, x.stride(0), r, ptr(od), o0, n, K, ptr(d2), None)
        call("ebsd_nlpar_average", ptr(x), hs, ws, n_pix, x.stride(0), r, ptr(od), o0, n, K, ptr(w), int(o0 > 0),
             ptr(out2), n_pix, None)
    grid = x[:, :n_pix].double().view(hs, ws, n_pix)
    shifts = [_shift(grid, a, b) for a, b in off.tolist()]
    ref_d = torch.stack([(s - grid).square().sum(-1) for s in shifts], -1).view(hs * ws, K)
    ref_o = sum(s * w[:, i].double().view(hs, ws, 1) for i, s in enumerate(shifts)).view(hs * ws, n_pix)
    # FP32 sums of n_pix terms of at most 1 and of K weighted values below 1
    assert (d.double() - ref_d).abs().max() <= 4 * n_pix * 2.0 ** -24
    assert (out.double() - ref_o).abs().max() <= 2 * K * 2.0 ** -24
    assert torch.equal(d, d2)
    assert (out2.double() - ref_o).abs().max() <= 4 * K * 2.0 ** -24


def test_repeated_and_outside_offsets():
    from ebsdtorch_b200._capi import call, ptr

    hs, ws, n_pix, r = 6, 11, 40, 2
    x = torch.rand((hs * ws, n_pix), device=DEV)
    off = torch.tensor([[0, 0], [0, 1], [0, 1], [2, -2], [3, 0], [-1, 0], [2, -2], [0, -3]])
    od = off.to(device=DEV, dtype=torch.int32)
    d = torch.full((hs * ws, 8), -1.0, device=DEV)
    call("ebsd_nlpar_dists", ptr(x), hs, ws, n_pix, n_pix, r, ptr(od), 0, 8, 8, ptr(d), None)
    assert torch.isnan(d[:, 4]).all() and torch.isnan(d[:, 7]).all()
    assert (d[:, 0] == 0).all() and torch.equal(d[:, 1], d[:, 2]) and torch.equal(d[:, 3], d[:, 6])
    grid = x.double().view(hs, ws, n_pix)
    for i in (1, 3, 5):
        ref = (_shift(grid, *off[i].tolist()) - grid).square().sum(-1).view(-1)
        assert (d[:, i].double() - ref).abs().max() <= 4 * n_pix * 2.0 ** -24
    out = torch.zeros_like(x)
    wts = torch.rand((hs * ws, 2), device=DEV)
    bad = torch.tensor([[0, 0], [0, 3]], dtype=torch.int32, device=DEV)
    call("ebsd_nlpar_average", ptr(x), hs, ws, n_pix, n_pix, r, ptr(bad), 0, 2, 2, ptr(wts), 0, ptr(out), n_pix, None)
    assert torch.isnan(out).all()
