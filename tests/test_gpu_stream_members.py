"""Single linears on slab weights whose row blocks are shared by few and by many streams: the sums of up to four members and those of
more are fetched by different code. Operands are whole numbers whose sums are exact in fp32, so every order gives the same bits."""
import pytest
import torch

import quantforge_b200 as qf

pytestmark = pytest.mark.gpu


# 296 streams on 148 multiprocessors: 1 to 2, 2 to 3, 4 to 5, 5 to 6, 8 to 9 and 16 to 18 members a row block, and half row blocks
@pytest.mark.parametrize("epilogue", [qf.QF_EPI_NONE, qf.QF_EPI_SILU_MUL, qf.QF_EPI_RESIDUAL_ADD])
@pytest.mark.parametrize("M,N,K", [(12, 37888, 4096), (9, 18944, 8192), (17, 9536, 8192), (32, 7680, 8192), (15, 4736, 14336),
                                   (25, 2368, 28672)])
def test_members(M, N, K, epilogue):
    gen = torch.Generator(device="cuda").manual_seed(N + M)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = torch.ones(K // 128, N, dtype=torch.float16, device="cuda")
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen))
    # |x| <= 8 and weights to 15: partial sums below 8 * 15 * K < 2^24
    x = torch.randint(-8, 9, (M, K), device="cuda", generator=gen).half()
    want = (x.double() @ qf.dequant_w4(qw, sc, zr).double().t()).float()
    res = torch.randint(-1000, 1001, (M, N), device="cuda", generator=gen).float()
    slab = qf.prepack_gemv_slab(qw, sc, zr)
    y = qf.w4a16_linear(x, slab, out_dtype=torch.float32, epilogue=epilogue, residual=res)
    if epilogue == qf.QF_EPI_SILU_MUL:
        r = want.view(M, -1, 2, 8).double()
        gate, up = r[:, :, 0].reshape(M, -1), r[:, :, 1].reshape(M, -1)
        exact = gate / (1 + torch.exp(-gate)) * up
        # expf within 2 ulp, then a sum, a division and two products: 1e-6 of the value
        assert bool(((y.double() - exact).abs() <= 1e-6 * exact.abs() + 1e-30).all())
    else:
        assert torch.equal(y, want + res if epilogue == qf.QF_EPI_RESIDUAL_ADD else want)
    for _ in range(2):
        assert torch.equal(qf.w4a16_linear(x, slab, out_dtype=torch.float32, epilogue=epilogue, residual=res), y)
    assert qf.device_status() == 0
