"""The NLPAR average over some of a window's offsets: values at the other
offsets take no part, non-finite ones included."""

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


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("r,offsets", [(0, [(0, 0)]), (1, [(0, 0)]), (1, [(0, 0), (0, 1), (1, 0), (0, -1), (-1, 0)]),
                                       (3, [(0, 0), (3, -3), (-2, 1)]), (7, [(7, 7), (0, 0), (-7, 2)])])
@pytest.mark.parametrize("n_pix", [63, 64])
def test_other_offsets_take_no_part(bad, r, offsets, n_pix):
    from ebsdtorch_b200._capi import call, ptr

    hs, ws, K = 11, 19, len(offsets)
    g = torch.Generator().manual_seed(r + K)
    x = torch.rand((hs * ws, n_pix), generator=g)
    x[5 * ws + 9, n_pix // 2] = bad
    w = torch.rand((hs * ws, K), generator=g) + 0.1
    ref = sum(_shift(x.view(hs, ws, n_pix), a, b).double() * w[:, i].double().view(hs, ws, 1)
              for i, (a, b) in enumerate(offsets)).view(hs * ws, n_pix)
    xd, wd, od = x.to(DEV), w.to(DEV), torch.tensor(offsets, dtype=torch.int32, device=DEV)
    out, blocks = (torch.full((hs * ws, n_pix), -1.0, device=DEV) for _ in range(2))
    call("ebsd_nlpar_average_window", ptr(xd), hs, ws, n_pix, n_pix, r, ptr(od), K, ptr(wd), ptr(out), n_pix, None)
    for o in range(K):
        call("ebsd_nlpar_average", ptr(xd), hs, ws, n_pix, n_pix, r, ptr(od), o, 1, K, ptr(wd), int(o > 0),
             ptr(blocks), n_pix, None)
    finite = ref.isfinite()
    for got in (out.cpu().double(), blocks.cpu().double()):
        assert torch.equal(got.isfinite(), finite)
        # FP32 sums of K products of values below 1.1
        assert (got - ref)[finite].abs().max() <= 4 * K * 1.1 * 2.0 ** -24
