"""Where the activations of a chain of 9 to 32 rows come from: another linear's results whole (read row block by row block as they are
finished), a part of them or those of several (read when the step before is complete), or nothing that the launch writes. Bit for bit
against the tcgen05 kernel, one linear after the other."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import ops
from quantforge_b200._lib import QF_PATH_GEMM

pytestmark = pytest.mark.gpu


def _pair(N, K, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 3 * N + K)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // 128, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen))
    return qf.prepack_gemv_slab(qw, sc, zr), (qf.prepack_w4(qw), sc, zr)


# (9 rows: five pairs of batch rows and eight members a row block, so some finish none)
@pytest.mark.parametrize("M,wide,dtype", [(9, 4096, torch.bfloat16), (16, 2816, torch.float16), (17, 4096, torch.float16), (32, 1408, torch.bfloat16)])
def test_sources(M, wide, dtype):
    def call(x, w, y, epilogue=qf.QF_EPI_NONE, residual=None):
        calls.append((x, w, y, epilogue, residual))

    runs = []
    for which in (0, 1):
        gen = torch.Generator(device="cuda").manual_seed(M)
        flat = torch.zeros(M * 4 * wide, device="cuda", dtype=dtype)
        at = lambda first, cols: flat[M * first:M * (first + cols)].view(M, cols)  # noqa: E731
        x = (torch.randn(M, wide, device="cuda", generator=gen) * 0.1).to(dtype)
        a, b, both, part = at(0, wide), at(wide, wide), at(0, 2 * wide), at(0, wide // 2 // 128 * 128)
        act, c = torch.zeros_like(x), torch.zeros_like(x)
        f32 = torch.zeros(M, wide, device="cuda")
        e = torch.zeros(M, wide // 2 // 128 * 128, device="cuda", dtype=dtype)
        late = [torch.zeros_like(x) for _ in range(2)]
        calls = []
        for i in range(3):
            w = lambda N, K: _pair(N, K, dtype, 10 * i + len(calls))[which]  # noqa: E731,B023
            call(x, w(wide, wide), a)                                     # nothing that the launch writes (but x, a step back)
            call(x, w(wide, wide), b)
            call(both, w(wide, 2 * wide), c)                              # two results
            call(c, w(2 * wide, wide), act, qf.QF_EPI_SILU_MUL)           # one, whole
            call(act, w(wide, wide), x, qf.QF_EPI_RESIDUAL_ADD, c)        # one, whole, two row blocks to a chunk
            call(part, w(e.shape[1], part.shape[1]), e)                   # part of one
            call(x, w(wide, wide), late[i % 2])
            call(x, w(wide, wide), f32)                                   # one, from several steps back; fp32 results
        runs.append((calls, [flat, x, act, c, f32, e] + late))
    (chain, got), (single, want) = runs
    for x, (qw, sc, zr), out, epilogue, residual in single:
        qf.w4a16_linear(x, qw, sc, zr, out=out, out_dtype=out.dtype, path=QF_PATH_GEMM, weight_layout=qf.QF_LAYOUT_INTERLEAVED,
                        epilogue=epilogue, residual=residual)
    start = [t.clone() for t in got]
    batch = ops.LinearBatch(chain)
    assert batch.launches() == 1
    for _ in range(4):
        for t, s in zip(got, start):
            t.copy_(s)
        batch.run()
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want))
    assert qf.device_status() == 0


# Launches in which nothing waits for the only phase, nothing is counted and nothing cleared, between launches that count: each leaves the
# counters as the next one needs them. Seven members a row block too, whose words are fetched in two goes.
@pytest.mark.parametrize("M", [9, 16, 17, 32])
def test_batches_without_waits_between_others(M):
    gen = torch.Generator(device="cuda").manual_seed(M)

    def linear(N, K):
        qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
        sc = (torch.rand(K // 128, N, device="cuda", generator=gen) * 0.003 + 0.0005).bfloat16()
        return qf.prepack_gemv_slab(qw, sc, qf.pack_zeros_u4(torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda",
                                                                           generator=gen)))
    x = torch.randn(M, 4096, device="cuda", generator=gen).bfloat16()
    e = lambda n: torch.zeros(M, n, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    first, second, third, wide = linear(4096, 4096), linear(4096, 4096), linear(1024, 4096), linear(512, 14336)
    a, b, c, d, act = e(4096), e(4096), e(1024), e(512), torch.randn(M, 14336, device="cuda", generator=gen).bfloat16()
    side = ops.LinearBatch([(x, first, a, qf.QF_EPI_NONE, None), (x, second, b, qf.QF_EPI_NONE, None), (x, third, c, qf.QF_EPI_NONE, None),
                            (act, wide, d, qf.QF_EPI_NONE, None)])
    row = ops.LinearBatch([(x, first, a, qf.QF_EPI_NONE, None), (a, second, b, qf.QF_EPI_NONE, None), (b, third, c, qf.QF_EPI_NONE, None),
                           (act, wide, d, qf.QF_EPI_NONE, None)])
    for batch in (side, row):
        assert batch.launches() == 1
    seen = {}
    for batch in (side, side, row, side, row, row, side):
        for y in (a, b, c, d):
            y.zero_()
        batch.run()
        got = [y.clone() for y in (a, b, c, d)]
        for u, v in zip(seen.setdefault(id(batch), got), got):
            assert torch.equal(u, v)
    assert torch.equal(seen[id(side)][0], seen[id(row)][0]) and torch.equal(seen[id(side)][3], seen[id(row)][3])
    assert qf.device_status() == 0
