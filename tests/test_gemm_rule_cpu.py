"""Which products take the long-K kernel's narrow tiles: at most one unit an SM
(148 where no GPU says otherwise), since their waves add up."""

import pytest
import torch

from ebsdtorch_b200._capi import DT_BF16, DT_E4M3, load


@pytest.mark.parametrize("m,n,k,dtype,narrow", [
    (32, 9, 1 << 20, DT_BF16, 1), (256, 2304, 4096, DT_BF16, 1), (128, 148 * 32, 2048, DT_BF16, 1),
    (128, 148 * 32 + 1, 2048, DT_BF16, 0), (2048, 1024, 10944, DT_BF16, 0), (1024, 794, 131072, DT_BF16, 0),
    (37 * 128, 128, 4096, DT_BF16, 1), (37 * 128, 129, 4096, DT_BF16, 0), (32, 9, 1984, DT_BF16, 0),
    (32, 9, 4096, DT_E4M3, 1), (32, 9, 3968, DT_E4M3, 0), (0, 9, 4096, DT_BF16, 0)])
def test_rule(m, n, k, dtype, narrow):
    if torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("written for 148 SMs")
    assert load().ebsd_gemm_nt_takes_narrow_tiles(m, n, k, dtype) == narrow
