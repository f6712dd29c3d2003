"""The BF16 GEMM of 65 to 128 columns on both sides of the line between tiles of 128 and of 256 rows (128-row
tiles times K splits against the number of SMs), with remainders of either tile.

Tolerance: as for the drained accumulators, 16 x 2^-23 a segment of 512 plus the float32 sums of at most 20
segments: 2e-6."""
import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_beyond", [0, 1])
@pytest.mark.parametrize("nr,K,splits,rest", [(65, 72, 1, 1), (128, 520, 1, 127), (100, 4608, 19, 128), (127, 10000, 4, 63)])
def test_both_tiles(nr, K, splits, rest, tiles_beyond):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    M = (sms // splits - 1 + tiles_beyond) * 128 + rest  # sms // splits tiles, or one more
    g = torch.Generator(device="cuda").manual_seed(nr + K)
    P = torch.rand((M, K), generator=g, device="cuda").to(torch.bfloat16)
    R = torch.rand((nr, K), generator=g, device="cuda").to(torch.bfloat16)
    got = ops.bf16_gemm_nt(P, R, k_splits=splits)
    torch.cuda.synchronize()
    assert _lib.take_gemm_timeout_count() == 0
    ref = P.double() @ R.double().T
    assert float(((got - ref).abs() / ref).max()) < 2e-6
