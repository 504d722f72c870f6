"""Dequantised weights at the edges of a block of rows and beyond the grid's second dimension, against the tensor statement."""
import pytest
import torch

import quantforge_b200 as qf

pytestmark = pytest.mark.gpu


def _want(qw, sc, z, group, dtype):
    N, K = qw.shape[0], qw.shape[1] * 2
    q = qf.unpack_int4(qw).view(N, K // group, group).float()
    w = (q - z.t().float().unsqueeze(-1)).to(dtype).float() * sc.t().float().unsqueeze(-1)
    return w.to(dtype).view(N, K)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,K,group", [(16, 128, 128), (32, 640, 128), (48, 512, 512), (80, 1152, 384), (112, 4224, 128), (1_048_592, 128, 128)])
def test_rows(N, K, group, dtype):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // group, N, device="cuda", generator=gen).abs() * 0.01).clamp_min(2.0 ** -14).to(dtype)
    z = torch.randint(0, 16, (K // group, N), dtype=torch.int8, device="cuda", generator=gen)
    assert torch.equal(qf.dequant_w4(qw, sc, z, group_size=group), _want(qw, sc, z, group, dtype))
    assert torch.equal(qf.dequant_w4(qw, sc, qf.pack_zeros_u4(z), group_size=group), _want(qw, sc, z, group, dtype))
    del qw, sc, z
    torch.cuda.empty_cache()  # a gigabyte of intermediate tensors
