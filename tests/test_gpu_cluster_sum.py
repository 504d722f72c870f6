"""Partial tiles of a cluster summed on chip: one round of sums and several, the last block's shorter share, every epilogue."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200._lib import QF_PATH_GEMM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [2, 3, 5, 7, 8])
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64])
def test_sums(M, split):
    dtype, N, K = (torch.bfloat16, torch.float16)[M % 2], 384, 4096
    gen = torch.Generator(device="cuda").manual_seed(M + split)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // 128, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen))
    x = torch.randn(M, K, device="cuda", generator=gen).to(dtype)
    res = torch.randn(M, N, device="cuda", generator=gen)
    ref = x.double() @ qf.dequant_w4(qw, sc, zr, group_size=128).double().t()
    pairs = ref.view(M, -1, 2, 8)
    gate, up = pairs[:, :, 0].reshape(M, -1), pairs[:, :, 1].reshape(M, -1)
    # fp32 sums of 4096 products: a few ulp of the largest partial sum. An error e in gate and up moves silu(gate) * up by at most
    # 1.1 e |up| + e |silu(gate)|; 16-bit results are rounded once more.
    e = 1e-4 * float(ref.pow(2).mean().sqrt())
    for epilogue, want, bound in ((qf.QF_EPI_NONE, ref, e), (qf.QF_EPI_RESIDUAL_ADD, ref + res.double(), e),
                                  (qf.QF_EPI_SILU_MUL, gate / (1 + torch.exp(-gate)) * up, 2.1 * e * float(ref.abs().max()))):
        for out_dtype in (torch.float32, dtype):
            residual = res.to(out_dtype) if epilogue == qf.QF_EPI_RESIDUAL_ADD else None
            exact = want if residual is None else ref + residual.double()
            y = qf.w4a16_linear(x, qf.prepack_w4(qw), sc, zr, out_dtype=out_dtype, weight_layout=qf.QF_LAYOUT_INTERLEAVED, path=QF_PATH_GEMM,
                                split_k=split, epilogue=epilogue, residual=residual)
            ulp = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[out_dtype]
            assert bool(((y.double() - exact).abs() <= bound + ulp * (exact.abs() + bound)).all())
            for _ in range(2):
                assert torch.equal(qf.w4a16_linear(x, qf.prepack_w4(qw), sc, zr, out_dtype=out_dtype, path=QF_PATH_GEMM, split_k=split,
                                                   weight_layout=qf.QF_LAYOUT_INTERLEAVED, epilogue=epilogue, residual=residual), y)
    assert qf.device_status() == 0
