"""CLAHE's passes over shapes that take their different branches: rows of whole
and of broken float4s, reflected padding, images staged in shared memory and
not, bins that are not a multiple of a warp. The min-max scalings use corrected
reciprocals and have to give what a division gives, bit for bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [(60, 60, 4, 4, 64), (61, 61, 4, 4, 64), (24, 40, 3, 5, 33), (9, 300, 2, 2, 2), (33, 17, 1, 1, 31),
          (200, 180, 8, 8, 257)]


def _clahe(x, h, w, sub, mm_in, mm_out, nb, gh, gw):
    from ebsdtorch_b200._capi import call, ptr

    out = torch.empty_like(x)
    call("ebsd_clahe", ptr(x), x.shape[0], h, w, x.stride(0), ptr(sub), mm_in, 40.0, nb, gh, gw, mm_out, ptr(out),
         out.stride(0), torch.cuda.current_stream().cuda_stream)
    return out


def _minmax(x):
    lo, hi = x.amin(dim=1, keepdim=True), x.amax(dim=1, keepdim=True)
    return (x - lo) / ((1e-4 + hi) - lo)


@pytest.mark.parametrize("h,w,gh,gw,nb", SHAPES)
@pytest.mark.parametrize("scale", [1e-30, 1.0, 200.0, 1e30])
def test_scalings_equal_divisions(h, w, gh, gw, nb, scale):
    g = torch.Generator(DEV).manual_seed(h * w + nb)
    x = torch.rand((5, h * w), device=DEV, generator=g) * scale
    x[1] = x[1, 0]  # a constant image
    sub = torch.rand(h * w, device=DEV, generator=g) * (0.1 * scale)
    plain = _clahe(_minmax(x - sub), h, w, None, 0, 0, nb, gh, gw)
    assert torch.equal(_clahe(x, h, w, sub, 1, 0, nb, gh, gw), plain)
    assert torch.equal(_clahe(x, h, w, sub, 1, 1, nb, gh, gw), _minmax(plain))


def test_rows_off_16_bytes():
    h, w = 20, 20
    g = torch.Generator(DEV).manual_seed(3)
    x = torch.rand((4, h * w), device=DEV, generator=g)
    ragged = torch.empty((4, h * w + 3), device=DEV)[:, 1:h * w + 1]
    ragged.copy_(x)
    sub = torch.rand(h * w + 1, device=DEV, generator=g)
    want = _clahe(x, h, w, sub[1:].clone(), 1, 1, 64, 4, 4)
    got = _clahe(ragged, h, w, sub[1:], 1, 1, 64, 4, 4)
    assert torch.equal(got, want)
