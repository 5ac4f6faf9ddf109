"""Products with a long K and few output tiles take narrow tiles: the same
bits as the wide tiles (an explicit split count keeps those), at the edges of
the staged rows and of the narrow columns, for an odd number of K steps, with
alpha and accumulation, and near float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m", [1, 32, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("n", [1, 9, 16, 17, 64, 257])
@pytest.mark.parametrize("k,lp", [(2048, "bf16"), (2112, "bf16"), (16384, "bf16"), (4096, "fp8"), (4224, "fp8")])
def test_narrow_tiles_give_the_same_bits(m, n, k, lp):
    from ebsdtorch_b200 import kernels
    from ebsdtorch_b200.kernels import LP_DTYPES, LP_TORCH, round_up

    g = torch.Generator(device=DEV).manual_seed(m * 1000 + n)
    dt = LP_DTYPES[lp]
    A = torch.randn((round_up(m, 128), k), generator=g, device=DEV).to(LP_TORCH[dt])
    B = torch.randn((round_up(n, 256), k), generator=g, device=DEV).to(LP_TORCH[dt])
    wide = B.shape[0] // 256
    outs = []
    for splits in (0, wide):
        out = torch.full((m, n + 3), 0.5, device=DEV)
        st = kernels.gemm_nt(A, B, out, alpha=0.25, m_valid=m, n_valid=n, splits=splits, lp_dtype=dt)
        st2 = kernels.gemm_nt(A, B, out, alpha=-2.0, accumulate=True, m_valid=m, n_valid=n, splits=splits,
                              lp_dtype=dt)
        assert int(st.item()) == 0 and int(st2.item()) == 0
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    assert (outs[0][:, n:] == 0.5).all()
    ref = -1.75 * A[:m].double() @ B[:n].double().T
    # FP32 accumulators that truncate: k / 16 additions of values up to about 4 sqrt(k)
    tol = 1.75 * (k / 16) * 2.0 ** -23 * 4 * k ** 0.5 + 1e-3
    assert (outs[0][:, :n].double() - ref).abs().max() < tol


@pytest.mark.parametrize("ldc", [64, 65, 96, 260])
def test_store_epilogue_alignments(ldc):
    from ebsdtorch_b200 import kernels

    g = torch.Generator(device=DEV).manual_seed(ldc)
    A = torch.randn((256, 64), generator=g, device=DEV).bfloat16()
    B = torch.randn((256, 64), generator=g, device=DEV).bfloat16()
    ref = A[:200].double() @ B.double().T
    for n in (1, 31, 33, min(ldc, 256)):
        for shift in (0, 1):
            flat = torch.zeros(200 * ldc + 1, device=DEV)
            out = flat[shift:shift + 200 * ldc].view(200, ldc)
            kernels.gemm_nt(A, B, out, m_valid=200, n_valid=min(n, ldc))
            kernels.gemm_nt(A, B, out, accumulate=True, m_valid=200, n_valid=min(n, ldc))
            assert (out[:, :n].double() - 2 * ref[:, :n]).abs().max() < 1e-3
            assert (out[:, n:] == 0).all()


def test_grouped_products_give_the_same_bits():
    from ebsdtorch_b200 import kernels

    g = torch.Generator(device=DEV).manual_seed(3)
    shapes = [(32, 9, 8192), (64, 288, 4096), (256, 40, 64), (129, 257, 128), (1, 1, 192), (128, 16, 2112)]
    prods, refs = [], []
    for m, n, k in shapes:
        A = torch.randn((-(-m // 128) * 128, k), generator=g, device=DEV).bfloat16()
        B = torch.randn((-(-n // 256) * 256, k), generator=g, device=DEV).bfloat16()
        ra, rb = -(-m // 16) * 16, -(-n // 16) * 16
        prods.append((A[:ra].view(ra, k // 64, 64).transpose(0, 1).contiguous(),
                      B[:rb].view(rb, k // 64, 64).transpose(0, 1).contiguous(), torch.zeros((m, n), device=DEV)))
        ref = torch.zeros((m, n), device=DEV)
        kernels.gemm_nt(A, B, ref, m_valid=m, n_valid=n, splits=B.shape[0] // 256)
        refs.append(ref)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.gemm_nt_group(prods, st)
    kernels.gemm_nt_group([], st)
    assert int(st.item()) == 0
    for (_, _, out), ref in zip(prods, refs):
        assert torch.equal(out, ref)
    with pytest.raises(Exception):
        kernels.gemm_nt_group(prods * 2, st)
