"""The kernels behind OrientationCNN.forward read FP32 pixels: patterns of
another type are converted first, and patterns on another device than the
weights are refused."""

import pytest
import torch

from ebsdtorch_b200 import learned
from ebsdtorch_b200.learned import OrientationCNN


class _Seen(Exception):
    pass


class _Conv:
    def __init__(self, device="cpu"):
        self.w = torch.zeros(1, device=device)

    def forward(self, x, *a, **k):
        raise _Seen(x)


def _net(device="cpu"):
    net = OrientationCNN.__new__(OrientationCNN)
    net.H, net.W, net.device, net.convs = 16, 16, torch.device(device), [_Conv(device)]
    return net


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16, torch.float64, torch.uint8,
                                   torch.uint16, torch.int32])
def test_kernels_get_fp32_pixels(monkeypatch, dtype, keep):
    cast = []

    def call(name, src, n, scale, dst, stream):
        assert name == "ebsd_cnn_scale_cast"
        cast.append((src, n, scale))

    monkeypatch.setattr(learned, "call", call)
    monkeypatch.setattr(learned, "ptr", lambda t: t)
    monkeypatch.setattr(learned, "_stream", lambda t: None)
    want = torch.arange(128 * 256).reshape(128, 16, 16) % 251
    x = want.to(dtype)
    with pytest.raises(_Seen) as seen:
        _net().forward(x, keep=keep)
    if keep:
        (src, n, scale), = cast
        assert n == src.numel() and scale == 1.0
    else:
        src, = seen.value.args
        assert not cast
    assert src.dtype == torch.float32 and src.is_contiguous() and torch.equal(src, want.float())


@pytest.mark.parametrize("keep", [False, True])
def test_patterns_elsewhere_than_the_weights_are_refused(keep):
    net = _net("meta")  # stands for another GPU of the same type
    net.device = torch.device("cpu")
    with pytest.raises(ValueError, match="network"):
        net.forward(torch.zeros((128, 16, 16)), keep=keep)
