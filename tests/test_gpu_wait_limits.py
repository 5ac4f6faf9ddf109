"""A wait that runs out in the convolution without columns and in the long-K
products: always reported, and the next call succeeds with the same results.

With a limit of 1 ns the epilogue gives up at the first poll that finds its
accumulator unfinished; every accumulator here takes hundreds of MMAs, and
a poll returns after about 200 ns. Nothing faults or hangs: the copies and MMAs in
flight complete before the kernel returns."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _check(run, out, status):
    from ebsdtorch_b200 import _capi

    lib = _capi.load()
    run()
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    good = out.clone()
    prev = lib.ebsd_set_wait_limit_ns(1)
    try:
        run()
        torch.cuda.synchronize()
    finally:
        assert lib.ebsd_set_wait_limit_ns(prev) == 1
    assert int(status.item()) == _capi.DEVICE_TIMEOUT
    status.zero_()
    out.zero_()
    run()
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and torch.equal(out, good)


@pytest.mark.parametrize("B", [1, 148 * 3])
def test_convolution(B):
    from ebsdtorch_b200._capi import call, ptr

    cin, cout, g = 1024, 256, torch.Generator(device=DEV).manual_seed(B)
    x = torch.randn((B, 16, 16, cin), device=DEV, generator=g).bfloat16()
    w = torch.randn((cout, 9 * cin), device=DEV, generator=g).bfloat16()
    out = torch.empty((B * 64, cout), dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    _check(lambda: call("ebsd_cnn_conv_tc", ptr(x), B, 16, 16, cin, ptr(w), 9 * cin, None, cout, 1, ptr(out), None,
                        ptr(status), None), out, status)


@pytest.mark.parametrize("m,n", [(32, 9), (256, 576)])
def test_long_products(m, n):
    from ebsdtorch_b200 import kernels

    k, g = 65536, torch.Generator(device=DEV).manual_seed(m)
    A = torch.randn((-(-m // 128) * 128, k), device=DEV, generator=g).bfloat16()
    B = torch.randn((-(-n // 256) * 256, k), device=DEV, generator=g).bfloat16()
    out, status = torch.empty((m, n), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    _check(lambda: kernels.gemm_nt(A, B, out, m_valid=m, n_valid=n, status=status), out, status)
    Ab, Bb = (t.view(-1, k // 64, 64).transpose(0, 1).contiguous() for t in (A, B))
    small = torch.empty((8, 8), device=DEV)
    _check(lambda: kernels.gemm_nt_group([(Ab, Bb, out), (Ab[:1], Bb[:1], small)], status), out, status)
