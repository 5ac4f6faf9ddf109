"""The convolution without columns against im2col + GEMM: the same bits, for
every channel pair it takes, odd and even sizes, output rows from one pixel to
a whole tile, tiles of several images and of part of one, and batches that do
not fill the last tile; and a wait that runs out is reported."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("cin,cout", [(32, 64), (64, 128), (128, 256), (256, 256)])
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (3, 2, 2), (5, 7, 5), (33, 8, 8), (9, 15, 15), (2, 30, 29), (130, 4, 4),
                                   (2, 33, 64), (1, 5, 255), (1, 3, 256)])
def test_same_bits_as_columns(cin, cout, B, H, W):
    from ebsdtorch_b200 import _capi
    from ebsdtorch_b200._capi import call, ptr
    from ebsdtorch_b200.learned import _Conv

    assert _capi.load().ebsd_cnn_conv_supported(cin, cout, W)
    gen = torch.Generator().manual_seed(cin + H)
    conv = _Conv(cin, cout, gen, torch.device(DEV))
    conv.b.copy_(torch.randn(cout, generator=gen) * 0.1)
    x = torch.randn((B, H, W, cin), generator=gen).to(DEV).bfloat16()
    M = B * ((H + 1) // 2) * ((W + 1) // 2)
    new16, old16 = (torch.full((M, cout), 3.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    new32, old32 = (torch.full((M, cout), 3.0, device=DEV) for _ in range(2))
    cols = conv._im2col(x, B, H, W)
    call("ebsd_cnn_conv_fwd", ptr(conv.w16), conv.w16.shape[0], ptr(cols), cols.shape[0], conv.K_pad, ptr(conv.b), cout,
         M, 1, ptr(old16), cout, ptr(old32), conv.fwd_splits, ptr(conv.status), None)
    for out32 in (new32, None):
        call("ebsd_cnn_conv_tc", ptr(x), B, H, W, cin, ptr(conv.w16), conv.K_pad, ptr(conv.b), cout, 1, ptr(new16),
             ptr(out32), ptr(conv.status), None)
        assert int(conv.status.item()) == 0
        assert torch.equal(new16, old16)
        new16.fill_(3.0)
    assert torch.equal(new32, old32)
    call("ebsd_cnn_conv_tc", ptr(x), B, H, W, cin, ptr(conv.w16), conv.K_pad, None, cout, 0, ptr(new16), ptr(new32),
         ptr(conv.status), None)
    w = conv.w16[:cout, :9 * cin].float().view(cout, 3, 3, cin).permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), w.double(), stride=2, padding=1)
    ref = ref.permute(0, 2, 3, 1).reshape(M, cout)
    assert (new32.double() - ref).abs().max() <= 1e-5 * ref.abs().max().clamp_min(1.0)


def test_a_wait_that_runs_out_is_reported():
    from ebsdtorch_b200 import _capi
    from ebsdtorch_b200._capi import DEVICE_TIMEOUT, call, ptr

    lib = _capi.load()
    x = torch.randn((64, 16, 16, 128), device=DEV).bfloat16()
    w = torch.randn((256, 1152), device=DEV).bfloat16()
    out = torch.empty((64 * 64, 256), dtype=torch.bfloat16, device=DEV)
    good = torch.empty_like(out)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(dst):
        call("ebsd_cnn_conv_tc", ptr(x), 64, 16, 16, 128, ptr(w), 1152, None, 256, 1, ptr(dst), None, ptr(st), None)

    run(good)
    torch.cuda.synchronize()
    assert int(st.item()) == 0
    lib.ebsd_set_wait_limit_ns(1)
    try:
        run(out)
        torch.cuda.synchronize()
        assert int(st.item()) in (0, DEVICE_TIMEOUT)
    finally:
        lib.ebsd_set_wait_limit_ns(0)
    st.zero_()
    run(out)
    torch.cuda.synchronize()
    assert int(st.item()) == 0 and torch.equal(out, good)


@pytest.mark.parametrize("B,H,W", [(128, 7, 9), (3, 16, 16), (1, 1, 1)])
@pytest.mark.parametrize("cout", [16, 32, 64])
def test_first_layer_rounds_fp32_pixels_as_the_cast_does(B, H, W, cout):
    from ebsdtorch_b200._capi import call, ptr

    g = torch.Generator().manual_seed(cout + H)
    x = torch.randn((B, H, W), generator=g).to(DEV)
    w = torch.randn((cout, 64), generator=g).to(DEV).bfloat16()
    b = torch.randn(cout, generator=g).to(DEV)
    M = B * ((H + 1) // 2) * ((W + 1) // 2)
    o16, p16 = (torch.zeros((M, cout), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    o32, p32 = (torch.zeros((M, cout), device=DEV) for _ in range(2))
    call("ebsd_cnn_conv_c1", ptr(x.bfloat16()), B, H, W, ptr(w), 64, ptr(b), cout, 1, ptr(o16), ptr(o32), None)
    call("ebsd_cnn_conv_c1_f32", ptr(x), B, H, W, ptr(w), 64, ptr(b), cout, 1, ptr(p16), ptr(p32), None)
    assert torch.equal(o16, p16) and torch.equal(o32, p32)
    ref = torch.nn.functional.conv2d(x.bfloat16().double().unsqueeze(1), w[:, :9].double().view(cout, 1, 3, 3),
                                     b.double(), stride=2, padding=1)
    ref = torch.relu(ref).permute(0, 2, 3, 1).reshape(M, cout)
    assert (o32.double() - ref).abs().max() <= 16 * 2.0 ** -24 * 9 * 16


@pytest.mark.parametrize("C", [1, 32, 64, 128])
@pytest.mark.parametrize("B,H,W", [(64, 1, 1), (16, 5, 7), (64, 6, 6), (8, 16, 15)])
def test_backward_operands(C, B, H, W):
    """Transposed columns, the fused ReLU gradient and the column gradient's
    scatter against torch, padding included."""
    from ebsdtorch_b200._capi import call, ptr

    Ho, Wo = (H + 1) // 2, (W + 1) // 2
    M = B * Ho * Wo
    g = torch.Generator().manual_seed(C + H)
    x = torch.randn((B, H, W, C), generator=g).to(DEV).bfloat16()
    pad = torch.nn.functional.pad(x, (0, 0, 1, 2, 1, 2))
    taps = [pad[:, ky:ky + 2 * Ho:2, kx:kx + 2 * Wo:2] for ky in range(3) for kx in range(3)]
    ref = torch.stack(taps, 3).reshape(M, 9 * C).t()
    out = torch.full((M // 64 + 1, 9 * C + 1, 64), 7.0, device=DEV).bfloat16()
    call("ebsd_cnn_im2col_t", ptr(x), B, H, W, C, ptr(out), 9 * C + 1, None)
    assert torch.equal(out[:-1, :9 * C].transpose(0, 1).reshape(9 * C, M), ref)
    assert (out[-1] == 7).all() and (out[:, 9 * C] == 7).all()
    dcols = torch.randn((M, 9 * C), generator=g).to(DEV)
    dx = torch.empty((B, H, W, C), device=DEV)
    call("ebsd_cnn_col2im", ptr(dcols), 9 * C, B, H, W, C, ptr(dx), None)
    acc = torch.zeros((B, H + 3, W + 3, C), device=DEV, dtype=torch.float64)
    for i in range(9):
        acc[:, i // 3:i // 3 + 2 * Ho:2, i % 3:i % 3 + 2 * Wo:2] += dcols[:, i * C:(i + 1) * C].double().view(B, Ho, Wo, C)
    assert (dx.double() - acc[:, 1:H + 1, 1:W + 1]).abs().max() <= 8 * 4 * 2.0 ** -23 * 4
    if C % 4:
        return
    dy = torch.randn((M, C), generator=g).to(DEV)
    act = torch.relu(torch.randn((M, C), generator=g)).to(DEV).bfloat16()
    ld16 = -(-C // 64) * 64
    want = torch.where(act.float() > 0, dy, torch.zeros_like(dy))
    for keep in (True, False):
        g16 = torch.full((M, ld16), 5.0, device=DEV).bfloat16()
        gT = torch.full((M // 64 + 1, C + 1, 64), 5.0, device=DEV).bfloat16()
        db = torch.full((C,), 5.0, device=DEV)
        call("ebsd_cnn_relu_grad_t", ptr(dy), ptr(act), M, C, ptr(g16) if keep else None, ld16, ptr(gT), C + 1,
             ptr(db), None)
        if keep:
            assert torch.equal(g16[:, :C], want.bfloat16()) and (g16[:, C:] == 0).all()
        assert torch.equal(gT[:-1, :C].transpose(0, 1).reshape(C, M), want.bfloat16().t())
        assert (gT[-1] == 5).all() and (gT[:, C] == 5).all()
        assert (db.double() - want.double().sum(0)).abs().max() <= M * 2.0 ** -23 * 4
