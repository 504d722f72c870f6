"""Linears right behind the work that writes their weights: a kernel of the stream that the linear may start beside."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200._lib import QF_PATH_GEMM, QF_PATH_GEMV

pytestmark = pytest.mark.gpu
N, K = 4096, 4096


def _call(kind, x, qw, sc, zr):
    if kind == "slab":
        return qf.w4a16_linear(x, qf.prepack_gemv_slab(qw, sc, zr))
    if kind == "tiled":
        return qf.w4a16_linear(x, qf.prepack_w4(qw, layout=qf.QF_LAYOUT_TILED), sc, zr, weight_layout=qf.QF_LAYOUT_TILED)
    return qf.w4a16_linear(x, qw, sc, zr, path=QF_PATH_GEMV if kind == "gemv" else QF_PATH_GEMM)


@pytest.mark.parametrize("kind,M", [("slab", 1), ("gemv", 1), ("gemm", 16), ("tiled", 100)])
def test_weights_written_by_the_previous_kernel(kind, M):
    """New codes and scales by elementwise kernels (and a prepack where the layout needs one), then the linear, with nothing
    in between; the same bits as with a synchronisation in between."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    base = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    s0 = (torch.rand(K // 128, N, device="cuda", generator=gen) * 0.01 + 0.001).bfloat16()
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen))
    x = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    qw, sc = base.clone(), s0.clone()
    _call(kind, x, qw, sc, zr)  # context and workspace
    got = []
    for i in range(8):
        torch.mul(s0, i + 1, out=sc)
        torch.bitwise_xor(base, 17 * i, out=qw)
        got.append(_call(kind, x, qw, sc, zr))
    for i, y in enumerate(got):
        q, s = base ^ (17 * i), s0 * (i + 1)
        torch.cuda.synchronize()
        want = _call(kind, x, q, s, zr)
        assert torch.equal(y, want)


@pytest.mark.parametrize("kind,M", [("slab", 1), ("gemv", 1), ("gemm", 16), ("tiled", 100)])
def test_captured_rows_of_linears(kind, M):
    """A captured row: linears behind a writer, behind each other, and behind a writer again. Replays read the weights that
    the same replay wrote."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    base = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.rand(K // 128, N, device="cuda", generator=gen) * 0.01 + 0.001).bfloat16()
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen))
    x = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    flip = torch.zeros(1, dtype=torch.int8, device="cuda")
    qw = [base.clone() for _ in range(3)]

    def row():
        for q in qw[:2]:
            torch.bitwise_xor(base, flip, out=q)
        y = [_call(kind, x, q, sc, zr) for q in qw[:2]]
        torch.bitwise_xor(base, flip + 1, out=qw[2])
        return y + [_call(kind, x, qw[2], sc, zr)]

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        row()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        outs = row()
    for v in (0, 51, -86):
        flip.fill_(v)
        g.replay()
        torch.cuda.synchronize()
        got = [y.clone() for y in outs]
        for y, f in zip(got, (v, v, v + 1)):
            q = base ^ f
            torch.cuda.synchronize()
            assert torch.equal(y, _call(kind, x, q, sc, zr))
