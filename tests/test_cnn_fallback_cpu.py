"""A convolution that the kernel without columns refuses (output rows of more
than 128 pixels) still makes its weight gradient's operand in the project's
kernel, from the activations."""

import pytest
import torch

from ebsdtorch_b200 import kernels, learned
from ebsdtorch_b200._capi import load


@pytest.mark.parametrize("cin,cout,W", [(32, 64, 258), (64, 128, 300), (256, 256, 257), (32, 64, 64)])
def test_operand_of_the_weight_gradient(monkeypatch, cin, cout, W):
    calls = []
    monkeypatch.setattr(learned, "call", lambda name, *a: calls.append((name, a)))
    monkeypatch.setattr(learned, "ptr", lambda t: t)
    monkeypatch.setattr(learned, "_stream", lambda t: None)
    monkeypatch.setattr(kernels, "gemm_nt", lambda *a, **k: calls.append(("gemm_nt", a)))
    assert bool(load().ebsd_cnn_conv_supported(cin, cout, W)) == (W <= 256)
    conv = learned._Conv(cin, cout, torch.Generator().manual_seed(0), torch.device("cpu"))
    x = torch.zeros((128, 1, W, cin), dtype=torch.bfloat16)
    keep, products = {}, []
    out, _, _, wo = conv.forward(x, 128, 1, W, keep)
    calls.clear()
    conv.backward(torch.zeros((128 * wo, cout)), keep, False, products)
    (name, args), = [c for c in calls if c[0].startswith("ebsd_cnn_im2col")]
    assert name == "ebsd_cnn_im2col_t" and args[0] is x and args[1:5] == (128, 1, W, cin)
    (gT, colsT, gw), = products
    assert args[5] is colsT and colsT.shape == (128 * wo // 64, 9 * cin, 64) and gw is conv.gw
