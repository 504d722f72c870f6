"""Batched calls (qf_w4a16_linear_batched) at the edges of what a chain takes."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import ops

pytestmark = pytest.mark.gpu


def _weights(N, K, dtype, seed, group=128, zeros=True):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // group, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // group, N), dtype=torch.int8, device="cuda", generator=gen)) if zeros else None
    return qw, sc, zr


def _slab(N, K, dtype, seed, group=128, zeros=True):
    return qf.prepack_gemv_slab(*_weights(N, K, dtype, seed, group, zeros), group_size=group)


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


def _same(a, b):
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))


@pytest.mark.parametrize("M,dtype", [(1, torch.bfloat16), (5, torch.float16), (8, torch.bfloat16)])
@pytest.mark.parametrize("special", [False, True])
def test_output_types_groups_zeros_and_special_values(M, dtype, special):
    """A chain of up to 8 rows has the bits of its linears one by one."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, 1024, device="cuda", generator=gen).to(dtype)
    if special:
        x[0, 5], x[0, 700], x[-1, 130], x[-1, 131] = float("inf"), float("inf"), float("nan"), float("-inf")
    calls = []
    for i in range(6):
        group, zeros = (128, 512, 1024)[i % 3], i % 2 == 0
        y, z = (torch.empty(M, 1024, device="cuda", dtype=t) for t in (dtype, torch.float32))
        calls += [(x, _slab(1024, 1024, dtype, i, group, zeros), y, qf.QF_EPI_NONE, None),
                  (x, _slab(1024, 1024, dtype, 50 + i, group, zeros), z, qf.QF_EPI_RESIDUAL_ADD, torch.ones_like(z)),
                  (y, _slab(1024, 1024, dtype, 90 + i, group, not zeros), torch.empty_like(z), qf.QF_EPI_NONE, None)]
        x = y
    batch = ops.LinearBatch(calls)
    assert batch.launches() == 1
    batch.run()
    got = [c[2].clone() for c in calls]
    for xi, w, out, epilogue, residual in calls:
        qf.w4a16_linear(xi, w, out=out, out_dtype=out.dtype, epilogue=epilogue, residual=residual)
    assert all(_same(c[2], g) for c, g in zip(calls, got))
    assert special == any(bool(g.isnan().any()) for g in got) and qf.device_status() == 0


def test_special_values_above_8_rows():
    """The bits of the tcgen05 kernel on interleaved weights; rows without special values are finite."""
    M, dtype = 11, torch.bfloat16
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, 1024, device="cuda", generator=gen).to(dtype)
    x[2, 5], x[4, 700], x[4, 701] = float("nan"), float("inf"), float("-inf")
    calls, want = [], []
    for i in range(4):
        qw, sc, zr = _weights(1024, 1024, dtype, i)
        calls.append((x, qf.prepack_gemv_slab(qw, sc, zr), torch.empty(M, 1024, device="cuda"), qf.QF_EPI_NONE, None))
        want.append(qf.w4a16_linear(x, qf.prepack_w4(qw), sc, zr, out_dtype=torch.float32, path=qf.QF_PATH_GEMM,
                                    weight_layout=qf.QF_LAYOUT_INTERLEAVED))
    batch = ops.LinearBatch(calls)
    assert batch.launches() == 1
    batch.run()
    clean = [m for m in range(M) if m not in (2, 4)]
    for (_, _, out, _, _), w in zip(calls, want):
        assert _same(out, w) and bool(out[clean].isfinite().all()) and bool(out[2].isnan().all())
    assert qf.device_status() == 0


@pytest.mark.parametrize("M", [1, 12])
def test_two_streams(M):
    """Chains on two streams at once: each has a workspace of its own."""
    dtype, batches, want = torch.bfloat16, [], []
    for s in range(2):
        h = [torch.randn(M, 1024, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)).to(dtype)]
        calls = []
        for i in range(12):
            h.append(torch.empty_like(h[0]))
            calls += [(h[i], _slab(1024, 1024, dtype, 40 * s + i), h[i + 1], qf.QF_EPI_NONE, None),
                      (h[i], _slab(1024, 1024, dtype, 40 * s + 20 + i), torch.empty_like(h[0]), qf.QF_EPI_NONE, None)]
        batch = ops.LinearBatch(calls)
        assert batch.launches() == 1
        batch.run()
        batches.append((batch, [c[2] for c in calls]))
        want.append([c[2].clone() for c in calls])
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in streams:
        with torch.cuda.stream(s):
            batches[0][0].run()  # makes the stream's workspace
        s.synchronize()
    for _ in range(20):
        for s, (batch, _) in zip(streams, batches):
            with torch.cuda.stream(s):
                batch.run()
    torch.cuda.synchronize()
    for (_, outs), w in zip(batches, want):
        assert all(torch.equal(o, v) for o, v in zip(outs, w))
    assert qf.device_status() == 0
