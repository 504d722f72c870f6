"""Batched calls (qf_w4a16_linear_batched) at the edges of what a chain takes."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import ops

pytestmark = pytest.mark.gpu


def _slab(N, K, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // 128, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen))
    return qf.prepack_gemv_slab(qw, sc, zr, group_size=128)


def test_no_rows_no_launch():
    x = torch.empty(0, 512, device="cuda", dtype=torch.float16)
    calls = [(x, _slab(512, 512, torch.float16, i), torch.empty_like(x), qf.QF_EPI_NONE, None) for i in range(20)]
    batch = ops.LinearBatch(calls)
    before = qf.launch_count()
    assert batch.launches() == 0
    batch.run()
    assert qf.launch_count() == before and qf.device_status() == 0


@pytest.mark.parametrize("M", [1, 8, 9, 24])
def test_a_result_over_weights_that_an_earlier_linear_reads(M):
    """Pairs of linears of the same activations; the second one's result goes over the weights of the first."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, 2048, device="cuda", generator=gen).to(torch.bfloat16)
    calls, want = [], []
    for i in range(8):
        first, second = _slab(2048, 2048, torch.bfloat16, i), _slab(2048, 2048, torch.bfloat16, 100 + i)
        over = first.blob[8192:8192 + M * 4096].view(torch.bfloat16).view(M, 2048)
        want += [qf.w4a16_linear(x, first), qf.w4a16_linear(x, second)]
        calls += [(x, first, torch.empty_like(over), qf.QF_EPI_NONE, None), (x, second, over, qf.QF_EPI_NONE, None)]
    torch.cuda.synchronize()
    batch = ops.LinearBatch(calls)
    assert batch.launches() == 1
    batch.run()
    for (_, _, out, _, _), w in zip(calls, want):
        # above 8 rows a chain adds in another order than the linear by itself: a rounding of bf16, 2^-8 of a value
        assert float((out.float() - w.float()).abs().max()) <= (0.0 if M <= 8 else 2.0 ** -7 * float(w.float().abs().max()))
    assert qf.device_status() == 0
