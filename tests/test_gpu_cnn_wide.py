"""Gradients of a convolution whose output rows are wider than the kernel
without columns takes, against float64 from the same bf16 operands."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("cin,cout,H,W", [(32, 64, 2, 258), (64, 128, 1, 259)])
def test_backward_of_a_wide_layer(cin, cout, H, W):
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200._capi import load
    from ebsdtorch_b200.learned import _Conv

    assert not load().ebsd_cnn_conv_supported(cin, cout, W)
    B, gen = 128, torch.Generator().manual_seed(W)
    conv = _Conv(cin, cout, gen, torch.device(DEV))
    x = torch.randn((B, H, W, cin), generator=gen).to(DEV).bfloat16()
    keep, products = {}, []
    out, _, ho, wo = conv.forward(x, B, H, W, keep)
    dout = torch.randn((B * ho * wo, cout), generator=gen).to(DEV)
    conv.backward(dout, keep, False, products)
    kernels.gemm_nt_group(products, conv.status)
    g = torch.where(out.float() > 0, dout, torch.zeros_like(dout))
    g64 = g.bfloat16().double().view(B, ho, wo, cout).permute(0, 3, 1, 2)
    w = torch.zeros((cout, cin, 3, 3), dtype=torch.float64, device=DEV, requires_grad=True)
    torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), w, stride=2, padding=1).backward(g64)
    ref = w.grad.permute(0, 2, 3, 1).reshape(cout, 9 * cin)
    # the accumulators truncate: at most 2^-23 of the sum's size a step of 16 pixels
    m = B * ho * wo
    assert (conv.gw.double() - ref).abs().max() <= 2.0 ** -23 * (m / 16) * ref.abs().max()
    assert (conv.gb.double() - g.double().sum(0)).abs().max() <= m * 2.0 ** -23 * 4
    assert int(conv.status.item()) == 0
