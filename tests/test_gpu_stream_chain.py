"""Streaming kernels (unpack, dequant, quantise, packs, prepacks) start while their predecessor on the stream still runs: a chain
of them, each reading what the one before wrote into reused buffers, gives the bits of the same calls one at a time."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu


def _chain(w, group, sync):
    def step(t):
        if sync:
            torch.cuda.synchronize()
        return t
    codes, scales, zeros = step(quantize_w4(w, group))
    qw = step(qf.pack_int4(codes))
    qz = step(qf.pack_zeros_u4(zeros))
    dense = step(qf.dequant_w4(qw, scales, qz, group_size=group))
    slab = step(qf.prepack_gemv_slab(qw, scales, qz, group_size=group))
    tiled = step(qf.prepack_w4(qw, layout=qf.QF_LAYOUT_TILED))
    back = step(qf.unpack_gemv_slab(slab))
    codes2 = step(qf.unpack_int4(back))
    return codes, scales, zeros, qw, qz, dense, slab.blob, tiled, codes2


@pytest.mark.parametrize("N,K,group", [(128, 128, 128), (256, 4096, 128), (2048, 4096, 128), (4096, 4096, 256), (384, 640, 640)])
def test_chain_equals_single_calls(N, K, group):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(N + K)
    w = [(torch.randn(N, K, device=dev, generator=gen) * 0.02).to(torch.bfloat16) for _ in range(3)]
    want = [[t.clone() for t in _chain(x, group, True)] for x in w]
    live = torch.empty_like(w[0])
    for _ in range(5):
        for x, ref in zip(w, want):
            live.copy_(x)  # the weight is written right before it is read, the temporaries are freed and handed out again
            got = _chain(live, group, False)
            for a, b in zip(got, ref):
                assert torch.equal(a, b)
            assert torch.equal(got[0], got[-1].view(N, K))


def test_chain_in_a_graph():
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(5)
    w = [(torch.randn(1024, 2048, device=dev, generator=gen) * 0.02).to(torch.bfloat16) for _ in range(2)]
    want = [[t.clone() for t in _chain(x, 128, True)] for x in w]
    live = w[0].clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = _chain(live, 128, False)
    for _ in range(5):
        for x, ref in zip(w, want):
            live.copy_(x)
            g.replay()
            for a, b in zip(got, ref):
                assert torch.equal(a, b)
