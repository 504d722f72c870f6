"""Chains of linears of up to 8 rows on slab weights in one launch (qf_w4a16_linear_batched): the bits of the linears one by one."""
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


def _chain(M, widths, fan, layers, dtype, seed=0):
    """Layers of: `fan` linears of the state, one with the residual from the first of them, SiLU * mul, and back with the residual.
    Widths: state, fan outputs, inner."""
    H, A, F = widths
    gen = torch.Generator(device="cuda").manual_seed(seed + M)
    empty = lambda n: torch.zeros(M, n, device="cuda", dtype=dtype)  # noqa: E731
    x = (torch.randn(M, H, device="cuda", generator=gen) * 0.1).to(dtype)
    calls, h = [], x
    b = {"fan": [empty(A) for _ in range(fan)], "o": empty(H), "act": empty(F), "h": [empty(H), empty(H)]}
    for i in range(layers):
        s = 10 * i
        calls += [(h, _slab(A, H, dtype, s + f), b["fan"][f], qf.QF_EPI_NONE, None) for f in range(fan)]
        calls += [(b["fan"][0], _slab(H, A, dtype, s + 6), b["o"], qf.QF_EPI_RESIDUAL_ADD, h),
                  (b["o"], _slab(2 * F, H, dtype, s + 7), b["act"], qf.QF_EPI_SILU_MUL, None),
                  (b["act"], _slab(H, F, dtype, s + 8), b["h"][i & 1], qf.QF_EPI_RESIDUAL_ADD, b["o"])]
        h = b["h"][i & 1]
    return calls


def _outputs(calls):
    seen = {}
    for _, _, out, _, _ in calls:
        seen[out.data_ptr()] = out
    return list(seen.values())


# one unit a block and many; half pairs; K of one chunk and of an odd number; grids of one, two and four blocks per SM; 1 to 3 side by
# side; more linears than a launch takes; all of the ring's row pitches
@pytest.mark.parametrize("M,widths,fan,layers,dtype", [
    (1, (1024, 512, 1408), 3, 3, torch.bfloat16), (2, (128, 128, 384), 2, 4, torch.float16), (3, (1152, 384, 640), 1, 5, torch.bfloat16),
    (5, (2048, 2048, 5632), 1, 4, torch.bfloat16), (8, (3072, 3072, 8192), 1, 2, torch.float16), (1, (1664, 128, 24832), 2, 3, torch.float16),
    (8, (256, 256, 256), 3, 30, torch.bfloat16), (4, (4096, 1024, 14336), 3, 3, torch.bfloat16), (7, (1920, 5760, 128), 2, 4, torch.float16)])
def test_bits_of_the_single_calls(M, widths, fan, layers, dtype):
    calls = _chain(M, widths, max(fan, 2), layers, dtype)  # linears of which each waits for the one before it are no chain
    batch = ops.LinearBatch(calls)
    for x, w, out, epilogue, residual in calls:
        qf.w4a16_linear(x, w, out=out, out_dtype=out.dtype, epilogue=epilogue, residual=residual)
    want = [o.clone() for o in _outputs(calls)]
    assert float(want[-1].float().abs().max()) > 0 and bool(torch.isfinite(want[-1].float()).all())
    assert batch.launches() <= -(-len(calls) // ops.CHAIN_LINEARS)
    for _ in range(3):  # counters and partial sums are left as they were found
        for o in _outputs(calls):
            o.fill_(float("nan"))
        batch.run()
        assert all(torch.equal(o, w) for o, w in zip(_outputs(calls), want))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        batch.run()
    for o in _outputs(calls):
        o.zero_()
    g.replay()
    assert all(torch.equal(o, w) for o, w in zip(_outputs(calls), want))
    assert qf.device_status() == 0


def test_what_goes_one_by_one():
    """Few linears, large ones, and rows that differ: no chain, the same results."""
    for M, widths, layers, launches in ((1, (1024, 512, 1408), 1, 4), (1, (5888, 5888, 6400), 2, 8)):
        calls = _chain(M, widths, 1, layers, torch.bfloat16)
        batch = ops.LinearBatch(calls)
        assert batch.launches() == launches
        for x, w, out, epilogue, residual in calls:
            qf.w4a16_linear(x, w, out=out, out_dtype=out.dtype, epilogue=epilogue, residual=residual)
        want = [o.clone() for o in _outputs(calls)]
        batch.run()
        assert all(torch.equal(o, w) for o, w in zip(_outputs(calls), want))
    a, b = _chain(1, (1024, 512, 1408), 3, 3, torch.bfloat16), _chain(2, (1024, 512, 1408), 3, 3, torch.bfloat16)
    assert ops.LinearBatch(a + b).launches() == 2
