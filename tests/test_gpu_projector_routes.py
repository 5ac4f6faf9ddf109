"""The projector's two routes, the gather table and the four plain gathers:
the same rows bit for bit, and both the oracle's, at the edges of the launch
rule (row lengths around the thread counts and the 6,656-pixel switch) and of
the image (one pixel high or wide)."""

import numpy as np
import pytest
import torch

from oracle import di_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(h, w, n_pix, n_rows, seed):
    rng = np.random.default_rng(seed)
    mp = torch.from_numpy(rng.random((h, w))).float()
    rays = rng.standard_normal((n_pix, 3))
    rays /= np.linalg.norm(rays, axis=1, keepdims=True)
    q = rng.standard_normal((n_rows, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return mp, torch.from_numpy(rays).float(), torch.from_numpy(q).float()


@pytest.mark.parametrize("h,w", [(1, 1), (1, 7), (5, 1), (2, 2), (33, 66)])
@pytest.mark.parametrize("n_pix,n_rows", [(1, 3), (255, 2), (513, 2), (6656, 2), (6657, 2)])
def test_routes_agree(h, w, n_pix, n_rows):
    from ebsdtorch_b200 import _capi, kernels
    from ebsdtorch_b200.kernels import RowBuffers

    mp, rays, q = _case(h, w, n_pix, n_rows, h * 1000 + n_pix)
    a, b = (torch.full((n_rows, n_pix), -7.0, device=DEV) for _ in range(2))
    args = (mp.to(DEV), rays.t().contiguous().to(DEV), q.to(DEV))
    plain = RowBuffers(f32=a)
    _capi.call("ebsd_project_dictionary", _capi.ptr(args[0]), h, w, _capi.ptr(args[1]), n_pix, _capi.ptr(args[2]),
               n_rows, 0, *plain.args(n_pix), None)
    torch.cuda.synchronize()
    kernels.project(*args, RowBuffers(f32=b), subtract_mean=False, quads=kernels.sampling_quads(args[0]))
    assert torch.equal(a, b)
    ref = O.project_patterns(mp.numpy().astype(np.float64), rays.numpy().astype(np.float64),
                             q.numpy().astype(np.float64))
    # a coordinate is off by at most about 8 roundings of a value below the
    # image size, more near the poles (1 - |z| of FP32 z): sqrt(2^-23) of a
    # quarter of the width there; values differ by at most 1 a pixel
    off = np.abs(b.cpu().numpy() - ref)
    assert off.max() <= np.sqrt(2.0 ** -23) * max(h, w) / 4 + 1e-6
    assert np.median(off) <= 8 * 2.0 ** -24 * max(h, w)


@pytest.mark.parametrize("dtype", [torch.float32, torch.uint16, torch.uint8, torch.float16])
@pytest.mark.parametrize("shape,shift", [((1, 1), 0), ((3, 5), 0), ((61, 61), 0), ((64, 64), 0), ((64, 64), 1),
                                         ((64, 65), 0), ((128, 128), 0), ((128, 129), 0)])
@pytest.mark.parametrize("lp", ["bf16", "fp8"])
def test_preparation_at_the_edges_of_its_rules(dtype, shape, shift, lp):
    """Row lengths at the thread-count switches and not multiples of 4 or 8,
    a base `shift` values off the vector alignment, both low-precision types:
    against float64, and the padding of the low-precision rows zero."""
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200.kernels import LP_DTYPES, LP_KMULT, LP_TORCH, RowBuffers, round_up

    h, w = shape
    n, n_pix, dt = 3, h * w, LP_DTYPES[lp]
    g = torch.Generator().manual_seed(n_pix)
    vals = torch.randint(0, 200, (n * n_pix + shift,), generator=g)
    flat = vals.to(torch.int32).to(dtype) if dtype in (torch.uint16, torch.uint8) else vals.to(dtype)
    x = flat.to(DEV)[shift:].view(n, h, w)
    kp = round_up(n_pix, LP_KMULT[dt])
    f32 = torch.empty((n, n_pix), device=DEV)
    low = torch.full((n, kp), 3.0, device=DEV).to(LP_TORCH[dt])
    norm, scale = torch.empty(n, device=DEV), torch.ones(n, device=DEV)
    kernels.prep_patterns(x, RowBuffers(f32=f32, lp=low, lp_dtype=dt, norm=norm, lp_scale=scale))
    ref = vals[shift:].double().view(n, n_pix)
    ref = ref - ref.mean(1, keepdim=True)
    # values below 200: mean and difference each round once
    assert (f32.cpu().double() - ref).abs().max() <= 2 * 200 * 2.0 ** -24
    rn = ref.norm(dim=1)
    assert (norm.cpu().double() - rn).abs().max() <= 1e-6 * rn.max() + 1e-4
    if n_pix > 1:
        unit = low.float().cpu().double()[:, :n_pix] * (scale.cpu().double()[:, None] if lp == "fp8" else 1.0)
        want = ref / rn[:, None]
        assert (unit - want).abs().max() <= (2.0 ** -8 if lp == "bf16" else 2.0 ** -3) * want.abs().max()
    assert torch.all(low.float()[:, n_pix:] == 0)
