"""Linears right behind the library's own kernels that write their weights, scales and zero points: these let their successor in
early, so a linear may be resident while they still write. Buffers are written anew each time; the bits are those of the same
calls with a synchronisation after each."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200._lib import QF_PATH_GEMM, QF_PATH_GEMV
from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu

# kind of weights, rows of activations, N (GEMV: not a multiple of 128 as well), K, group size
CASES = [("gemv", 1, 4096, 4096, 128), ("gemv", 3, 1040, 1024, 128), ("gemv", 8, 528, 2048, 2048), ("slab", 1, 4096, 4096, 128),
         ("slab", 5, 1024, 2048, 256), ("gemm", 16, 2048, 4096, 128), ("gemm", 130, 1024, 1024, 1024), ("interleaved", 40, 1024, 2048, 128),
         ("tiled", 4, 4096, 2048, 128)]


def _chain(kind, w, x, group, zeros_u4, sync):
    def step(t):
        if sync:
            torch.cuda.synchronize()
        return t
    codes, scales, zeros = step(quantize_w4(w, group))
    qw = step(qf.pack_int4(codes))
    if zeros_u4:
        zeros = step(qf.pack_zeros_u4(zeros))
    if kind == "slab":
        return step(qf.w4a16_linear(x, step(qf.prepack_gemv_slab(qw, scales, zeros, group_size=group))))
    if kind in ("gemv", "gemm"):
        return step(qf.w4a16_linear(x, qw, scales, zeros, group, path=QF_PATH_GEMV if kind == "gemv" else QF_PATH_GEMM))
    layout = qf.QF_LAYOUT_TILED if kind == "tiled" else qf.QF_LAYOUT_INTERLEAVED
    return step(qf.w4a16_linear(x, step(qf.prepack_w4(qw, layout=layout)), scales, zeros, group, weight_layout=layout))


def _inputs(M, N, K, dtype):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    # weights whose scales differ by powers of two: a stale scale is not within rounding of the right one
    ws = [(torch.randn(N, K, device="cuda", generator=gen) * 0.02 * 4.0 ** i).to(dtype) for i in range(3)]
    return ws, torch.randn(M, K, device="cuda", generator=gen).to(dtype)


@pytest.mark.parametrize("zeros_u4", [True, False])
@pytest.mark.parametrize("kind,M,N,K,group", CASES)
def test_linear_behind_the_writers(kind, M, N, K, group, zeros_u4):
    ws, x = _inputs(M, N, K, torch.bfloat16)
    want = [_chain(kind, w, x, group, zeros_u4, True).clone() for w in ws]
    live = torch.empty_like(ws[0])
    got = []
    for _ in range(4):
        for w in ws:
            live.copy_(w)
            got.append(_chain(kind, live, x, group, zeros_u4, False))
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 3])


@pytest.mark.parametrize("kind,M,N,K,group", CASES)
def test_linear_behind_the_writers_in_a_graph(kind, M, N, K, group):
    ws, x = _inputs(M, N, K, torch.float16)
    want = [_chain(kind, w, x, group, True, True).clone() for w in ws]
    live = ws[0].clone()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        _chain(kind, live, x, group, True, False)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        y = _chain(kind, live, x, group, True, False)
        z = _chain(kind, live, x, group, True, False)  # the second round's kernels follow a linear
    for _ in range(3):
        for w, ref in zip(ws, want):
            live.copy_(w)
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, ref) and torch.equal(z, ref)
