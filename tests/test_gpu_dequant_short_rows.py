"""Dequantised weights of one or two groups a row, of which a block takes 32 rows instead of 16 from a number of rows on: both sides of
that number, both ends of a block, and more blocks than the grid's second dimension holds, against the tensor statement."""
import ctypes

import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import _lib, ops
from test_gpu_dequant_rows import _want

pytestmark = pytest.mark.gpu


def _check(N, K, dtype, zeros):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.rand(K // 128, N, device="cuda", generator=gen) * 0.01 + 0.001).to(dtype)
    z = torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen) if zeros != "const" else \
        torch.full((K // 128, N), 8, dtype=torch.int8, device="cuda")
    zr = {"const": None, "i8": z, "u4": qf.pack_zeros_u4(z)}[zeros]
    assert torch.equal(qf.dequant_w4(qw, sc, zr, group_size=128), _want(qw, sc, z, 128, dtype))
    # (outputs that are aligned to 16 bytes only have a kernel of their own)
    out = torch.empty(N * K + 8, dtype=dtype, device="cuda")[8:].view(N, K)
    assert out.data_ptr() % 32 == 16
    half = _lib.QF_F16 if dtype == torch.float16 else _lib.QF_BF16
    d = _lib.LinearDesc(M=1, N=N, K=K, group_size=128, act_dtype=half, out_dtype=half, zero_const=8,
                        zero_mode={"const": _lib.QF_ZERO_CONST, "i8": _lib.QF_ZERO_I8, "u4": _lib.QF_ZERO_U4}[zeros])
    ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert _lib.load().qf_dequant_w4(ops._ctx(qw.device), ctypes.byref(d), ptr(qw), ptr(sc), ptr(zr), ptr(out),
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert torch.equal(out, _want(qw, sc, z, 128, dtype))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N", [32752, 32768, 32784, 32800, 65520, 65536, 65552])
@pytest.mark.parametrize("K,zeros", [(128, "const"), (256, "const"), (384, "const"), (128, "u4"), (128, "i8"), (256, "u4")])
def test_rows(N, K, zeros, dtype):
    _check(N, K, dtype, zeros)


@pytest.mark.parametrize("N,K,zeros", [(2_097_168, 128, "const"), (2_097_168, 128, "u4"), (1_048_592, 384, "i8")])
def test_more_blocks_than_the_second_dimension(N, K, zeros):
    _check(N, K, torch.float16, zeros)
    torch.cuda.empty_cache()  # gigabytes of intermediate tensors
