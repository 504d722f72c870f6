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
