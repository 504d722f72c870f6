"""Canonical weights whose rows are no multiple of 128, through the tcgen05 kernel: the last tile is cut short. Against float64 products
of the dequantised weights, at every length of that tile. (tests/test_ragged_plan.py has the rule that picks the kernel.)"""
import ctypes

import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import _lib
from quantforge_b200._lib import QF_PATH_GEMM, QF_PATH_GEMV

pytestmark = pytest.mark.gpu


def _inputs(M, K, N, zeros, group, dtype):
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // group, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    z = torch.randint(0, 16, (K // group, N), dtype=torch.int8, device="cuda", generator=gen)
    zr = {"u4": lambda: qf.pack_zeros_u4(z), "i8": lambda: z - 8, "const": lambda: None}[zeros]()
    return qw, sc, zr, torch.randn(M, K, device="cuda", generator=gen).to(dtype)


# the last tile has 16, 32, 48, 64, 80, 96, 112 rows, and is the only one at N = 112; one to eight splits on chip, splits through memory (65 rows
# and more), none
@pytest.mark.parametrize("M,K,N,zeros,group,dtype", [
    (3, 3968, 5136, "i8", 3968, torch.float16), (8, 8192, 1040, "i8", 128, torch.bfloat16), (5, 4096, 3104, "u4", 256, torch.float16),
    (16, 8192, 544, "u4", 128, torch.bfloat16), (17, 2048, 2128, "const", 2048, torch.float16), (33, 4096, 1120, "u4", 128, torch.bfloat16),
    (64, 2048, 20144, "i8", 128, torch.bfloat16), (100, 8192, 624, "const", 512, torch.float16), (200, 4096, 1136, "i8", 128, torch.bfloat16),
    (777, 1024, 4176, "const", 128, torch.float16), (300, 512, 28688, "i8", 512, torch.bfloat16),
    (24, 4096, 1088, "u4", 128, torch.float16), (128, 8192, 704, "u4", 128, torch.bfloat16), (32, 28672, 112, "i8", 128, torch.bfloat16)])
def test_last_tile(M, K, N, zeros, group, dtype):
    zero_mode = {"u4": _lib.QF_ZERO_U4, "i8": _lib.QF_ZERO_I8, "const": _lib.QF_ZERO_CONST}[zeros]
    half = _lib.QF_F16 if dtype == torch.float16 else _lib.QF_BF16
    d = _lib.LinearDesc(M=M, N=N, K=K, group_size=group, act_dtype=half, out_dtype=half, zero_mode=zero_mode, zero_const=8)
    planned = ctypes.c_int32()
    assert _lib.load().qf_w4a16_plan(ctypes.byref(d), ctypes.byref(planned), None) == 0 and planned.value == QF_PATH_GEMM
    qw, sc, zr, x = _inputs(M, K, N, zeros, group, dtype)
    ref = x.double() @ qf.dequant_w4(qw, sc, zr, group_size=group).double().t()
    rms = float(ref.pow(2).mean().sqrt())
    # one rounding of the output, and fp32 sums of up to 8192 products
    ulp, e = 2.0 ** (-8 if dtype == torch.bfloat16 else -11), 1e-4 * rms
    errors = {}
    for path in (_lib.QF_PATH_AUTO, QF_PATH_GEMV):
        guard = torch.full((M + 2, N), 7.0, device="cuda", dtype=dtype)
        y = qf.w4a16_linear(x, qw, sc, zr, group, out=guard[1:M + 1], path=path)
        assert bool(((y.double() - ref).abs() <= e + ulp * (ref.abs() + e)).all())
        assert bool((guard[0] == 7.0).all()) and bool((guard[M + 1] == 7.0).all())
        errors[path] = float((y.double() - ref).pow(2).mean().sqrt()) / rms
    assert errors[_lib.QF_PATH_AUTO] <= 1.001 * errors[QF_PATH_GEMV]
    # 32-bit results come from the other kernel
    f32 = [qf.w4a16_linear(x, qw, sc, zr, group, out_dtype=torch.float32, path=path) for path in (_lib.QF_PATH_AUTO, QF_PATH_GEMV)]
    assert torch.equal(*f32) and float((f32[0].double() - ref).abs().max()) < e
    y16 = qf.w4a16_linear(x, qw, sc, zr, group)
    first = y16.clone()
    for _ in range(3):
        assert torch.equal(qf.w4a16_linear(x, qw, sc, zr, group), first)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        qf.w4a16_linear(x, qw, sc, zr, group, out=y16)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        qf.w4a16_linear(x, qw, sc, zr, group, out=y16)
        qf.w4a16_linear(x, qw, sc, zr, group, out=y16)  # behind a linear
    y16.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y16, first) and qf.device_status() == 0


def test_scales_at_the_end_of_an_allocation_and_large_ones():
    # the last rows of the last group end where the tensors end; scales of 2^126 and more take another form of the converter
    M, K, N = 4, 4096, 2064
    qw, sc, zr, x = _inputs(M, K, N, "i8", 128, torch.bfloat16)
    qw[-3:], zr[:, -3:], sc[:, -3:] = 0x99 - 256, 8, 2.0 ** 126  # codes 9: weights of 2^126
    x = x * 2.0 ** -100
    y = qf.w4a16_linear(x, qw, sc, zr)
    ref = x.double() @ qf.dequant_w4(qw, sc, zr, group_size=128).double().t()
    e = 1e-4 * ref.pow(2).mean(0).sqrt() + 1e-4 * 2.0 ** -8 * ref.abs().amax(0)
    assert bool(((y.double() - ref).abs() <= e + 2.0 ** -8 * (ref.abs() + e)).all()) and float(ref[:, -3:].abs().min()) > 2.0 ** 20


@pytest.mark.parametrize("N", [5136, 5152])
def test_explicit_path_is_refused_as_before(N):
    qw, sc, zr, x = _inputs(4, 2048, N, "i8", 128, torch.float16)
    with pytest.raises(Exception, match="multiple of 128"):
        qf.w4a16_linear(x, qw, sc, zr, path=QF_PATH_GEMM)
