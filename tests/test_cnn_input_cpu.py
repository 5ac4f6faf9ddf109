"""What OrientationCNN.forward refuses before it hands a pointer to a kernel."""

import pytest
import torch

from ebsdtorch_b200.learned import OrientationCNN


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("shape,net_device", [((128, 15, 16), "cpu"), ((128, 16, 17), "cpu"), ((128, 2, 16, 16), "cpu"),
                                              ((127, 16, 16), "cpu"), ((128, 16, 16), "cuda")])
def test_refuses_patterns_that_do_not_fit(shape, net_device, keep):
    net = OrientationCNN.__new__(OrientationCNN)
    net.H, net.W, net.device, net.convs = 16, 16, torch.device(net_device), []
    with pytest.raises(ValueError):
        net.forward(torch.zeros(shape), keep=keep)
