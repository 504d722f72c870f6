"""tcgen05 kernel: the batch tile takes the width that the row count asks for (a multiple of 16, of 32 for a pair of blocks)."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200._lib import QF_PATH_GEMM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [48, 49, 65, 80, 81, 113, 129, 144, 145, 177, 209, 257, 270, 289, 513, 777])
@pytest.mark.parametrize("N", [256, 384])
@pytest.mark.parametrize("epilogue", ["none", "silu", "residual"])
def test_batch_tile_widths(M, N, epilogue):
    """Results as those of 64 rows at a time."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    K = 512
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.rand(K // 128, N, device="cuda", generator=gen) * 0.01 + 0.001).bfloat16()
    x = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=gen)
    epi = {"none": qf.QF_EPI_NONE, "silu": qf.QF_EPI_SILU_MUL, "residual": qf.QF_EPI_RESIDUAL_ADD}[epilogue]

    def call(a, r):
        return qf.w4a16_linear(a, qw, sc, None, out_dtype=torch.float32, epilogue=epi,
                               residual=r if epilogue == "residual" else None, path=QF_PATH_GEMM)

    y = call(x, res)
    want = torch.cat([call(x[i:i + 64].contiguous(), res[i:i + 64].contiguous()) for i in range(0, M, 64)])
    # fp32 sums of 512 products in another order: 512 * 2^-24 of the sum of magnitudes, which is below 22 rms of a sum; a
    # SiLU * mul output adds the errors of two of them, each times the other's value of at most 5 rms
    tol = 512 * 2.0 ** -24 * 22 * 10 * want.square().mean().sqrt()
    assert (y - want).abs().max() <= tol
