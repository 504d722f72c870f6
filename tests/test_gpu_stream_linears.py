"""The streaming tcgen05 kernel on slab weights: single linears that the size rule gives to it against an fp32 product with the
dequantised weights, and chains (qf_w4a16_linear_batched) bit for bit against the tcgen05 kernel on interleaved weights."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import ops
from quantforge_b200._lib import QF_PATH_GEMM

pytestmark = pytest.mark.gpu


def _weights(N, K, dtype, group=128, seed=0, scale=0.003):
    gen = torch.Generator(device="cuda").manual_seed(seed + N + K)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // group, N, device="cuda", generator=gen).abs() * scale).clamp_min(2.0 ** -14).to(dtype)
    zr = qf.pack_zeros_u4(torch.randint(0, 16, (K // group, N), dtype=torch.int8, device="cuda", generator=gen))
    return qw, sc, zr


def _x(M, K, dtype, seed=0, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed + M)
    return (torch.randn(M, K, device="cuda", generator=gen) * scale).to(dtype)


def _silu_mul(y):  # rows in eights of gate and up
    r = y.view(y.shape[0], -1, 2, 8)
    gate, up = r[:, :, 0].reshape(y.shape[0], -1), r[:, :, 1].reshape(y.shape[0], -1)
    return gate / (1 + torch.exp(-gate)) * up


# sizes that the rule gives to this kernel, half row blocks at the end, few and many members a row block; and some beyond its lines, which
# the streaming GEMV kernel serves (12 and 25 rows of short K, up to 8 rows of any size)
@pytest.mark.parametrize("M,N,K,dtype,group", [
    (9, 8256, 8192, torch.bfloat16, 128), (16, 2112, 28672, torch.float16, 256), (12, 17408, 4096, torch.float16, 128),
    (17, 6208, 8192, torch.bfloat16, 8192), (25, 24640, 2048, torch.float16, 128), (32, 1792, 28672, torch.bfloat16, 128),
    (3, 57344, 5760, torch.bfloat16, 128), (8, 11520, 28672, torch.float16, 128),
    (12, 34880, 4096, torch.float16, 128), (25, 81984, 1024, torch.bfloat16, 128)])
def test_single_linear(M, N, K, dtype, group):
    qw, sc, zr = _weights(N, K, dtype, group)
    slab, x = qf.prepack_gemv_slab(qw, sc, zr, group_size=group), _x(M, K, dtype)
    ref = x.float() @ qf.dequant_w4(qw, sc, zr, group_size=group).float().t()
    res = _x(M, N, torch.float32, seed=7)
    guard = torch.full((M + 2, N), 7.0, device="cuda")
    # fp32 sums of K products in two orders: a few ulp of the largest partial sum. An error e in gate and up moves
    # silu(gate) * up by at most 1.1 e |up| + e |silu(gate)|.
    e = 1e-4 * float(ref.pow(2).mean().sqrt())
    for epilogue, want, bound in ((qf.QF_EPI_NONE, ref, e), (qf.QF_EPI_RESIDUAL_ADD, ref + res, e),
                                  (qf.QF_EPI_SILU_MUL, _silu_mul(ref), 2.1 * e * float(ref.abs().max()))):
        out = guard[1:M + 1] if epilogue != qf.QF_EPI_SILU_MUL else None
        call = lambda o=None: qf.w4a16_linear(x, slab, out_dtype=torch.float32, out=o, epilogue=epilogue, residual=res)  # noqa: E731
        y = call(out)
        assert float((y - want).abs().max()) < bound
        first = y.clone()
        for _ in range(3):
            assert torch.equal(call(), first)
    assert bool((guard[0] == 7.0).all()) and bool((guard[M + 1] == 7.0).all())
    assert qf.device_status() == 0


def _layers(hidden, kv, ffn, n, dtype):
    """Weights of n layers as (slab, interleaved) pairs by name."""
    made = []
    for i in range(n):
        ly = {}
        for name, (N, K) in {"qkv": (hidden + 2 * kv, hidden), "o": (hidden, hidden), "gate_up": (2 * ffn, hidden), "down": (hidden, ffn)}.items():
            qw, sc, zr = _weights(N, K, dtype, seed=100 * i)
            ly[name] = (qf.prepack_gemv_slab(qw, sc, zr), (qf.prepack_w4(qw), sc, zr))
        made.append(ly)
    return made


def _buffers(M, hidden, kv, ffn, dtype):
    e = lambda n: torch.zeros(M, n, device="cuda", dtype=dtype)  # noqa: E731
    return {"h": _x(M, hidden, dtype, 1, 0.02), "attn": _x(M, hidden, dtype, 2, 0.02), "qkv": e(hidden + 2 * kv), "o": e(hidden),
            "act": e(ffn), "down": e(hidden)}


def _calls(layers, b, which):
    calls, h = [], b["h"]
    for ly in layers:
        calls += [(h, ly["qkv"][which], b["qkv"], qf.QF_EPI_NONE, None), (b["attn"], ly["o"][which], b["o"], qf.QF_EPI_RESIDUAL_ADD, h),
                  (b["o"], ly["gate_up"][which], b["act"], qf.QF_EPI_SILU_MUL, None),
                  (b["act"], ly["down"][which], b["down"], qf.QF_EPI_RESIDUAL_ADD, b["o"])]
        h = b["down"]
    return calls


def _one_by_one(calls):
    for x, (qw, sc, zr), out, epilogue, residual in calls:
        qf.w4a16_linear(x, qw, sc, zr, out=out, out_dtype=out.dtype, path=QF_PATH_GEMM, weight_layout=qf.QF_LAYOUT_INTERLEAVED,
                        epilogue=epilogue, residual=residual)


@pytest.mark.parametrize("M,hidden,kv,ffn,layers,dtype", [
    (9, 1024, 512, 2816, 3, torch.bfloat16), (16, 1152, 128, 1280, 2, torch.float16), (13, 4096, 1024, 14336, 2, torch.bfloat16),
    (17, 1024, 256, 5632, 2, torch.float16), (32, 2048, 512, 2048, 2, torch.bfloat16), (10, 512, 128, 1536, 30, torch.bfloat16),
    (9, 256, 128, 18944, 2, torch.float16), (24, 4096, 1024, 14336, 2, torch.bfloat16)])
def test_chain_is_the_tcgen05_kernel_bit_for_bit(M, hidden, kv, ffn, layers, dtype):
    made = _layers(hidden, kv, ffn, layers, dtype)
    want, got = _buffers(M, hidden, kv, ffn, dtype), _buffers(M, hidden, kv, ffn, dtype)
    _one_by_one(_calls(made, want, 1))
    batch = ops.LinearBatch(_calls(made, got, 0))
    before = qf.launch_count()
    batch.run()
    assert qf.launch_count() - before == -(-4 * layers // ops.CHAIN_LINEARS)
    assert all(torch.equal(want[k], got[k]) for k in want)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        batch.run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        batch.run()
    for _ in range(3):
        for k in ("qkv", "o", "act", "down"):
            got[k].zero_()
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(want[k], got[k]) for k in want)
    assert qf.device_status() == 0


@pytest.mark.parametrize("M", [1, 8, 9, 16, 33 - 1])
def test_batch_of_mixed_linears(M):
    """What a chain does not take (few rows, half row blocks, other rows in between) runs by itself, in order."""
    shapes = [(256, 512), (512, 256), (192, 512), (512, 256)]
    weights = [_weights(N, K, torch.float16, seed=i) for i, (N, K) in enumerate(shapes)]
    slabs = [qf.prepack_gemv_slab(*w) for w in weights]
    x, lone = _x(M, 512, torch.float16), _x(3, 512, torch.float16)
    outs = [torch.empty(m, N, device="cuda") if i in (2, 4) else torch.empty(m, N, device="cuda", dtype=torch.float16)
            for i, (m, N) in enumerate([(M, 256), (M, 512), (M, 192), (M, 512), (3, 256)])]
    calls = [(x, slabs[0], outs[0], qf.QF_EPI_NONE, None), (outs[0], slabs[1], outs[1], qf.QF_EPI_RESIDUAL_ADD, x),
             (outs[1], slabs[2], outs[2], qf.QF_EPI_NONE, None), (outs[0], slabs[3], outs[3], qf.QF_EPI_RESIDUAL_ADD, outs[1]),
             (lone, slabs[0], outs[4], qf.QF_EPI_NONE, None)]
    ops.LinearBatch(calls).run()
    for (xi, _, out, epilogue, residual), w in zip(calls, weights + weights[:1]):
        ref = xi.float() @ qf.dequant_w4(*w).float().t()
        if epilogue == qf.QF_EPI_RESIDUAL_ADD:
            ref = ref + residual.float()
        # the output's rounding, 2^-11 of a value, on top of the sums'
        tol = 1e-4 if out.dtype == torch.float32 else 4 * 2.0 ** -11
        assert float((out.float() - ref).abs().max() / ref.pow(2).mean().sqrt()) < tol
    assert qf.device_status() == 0


def test_results_that_become_weights_end_a_chain():
    """The second linear's blob lies in the buffer that the first one writes, so it must not be fetched ahead."""
    M, N, K = 16, 2176, 256
    slab = qf.prepack_gemv_slab(*_weights(N, K, torch.bfloat16))
    target = qf.prepack_gemv_slab(*_weights(128, 1024, torch.bfloat16, seed=5))
    # M * N bf16 outputs are as many bytes as the blob of 128 x 1024: 16 * 2176 * 2 = 2 * 8 * 4352
    alias = ops.SlabWeight(torch.zeros(M, N, device="cuda", dtype=torch.bfloat16).view(torch.uint8).view(-1), 128, 1024, 128, torch.bfloat16,
                           target.zero_mode, 8)
    assert alias.blob.numel() == target.blob.numel()
    out = alias.blob.view(torch.bfloat16).view(M, N)
    y = torch.empty(M, 128, device="cuda")
    before = qf.launch_count()
    ops.LinearBatch([(_x(M, K, torch.bfloat16), slab, out, qf.QF_EPI_NONE, None),
                     (_x(M, 1024, torch.bfloat16), alias, y, qf.QF_EPI_NONE, None)]).run()
    assert qf.launch_count() - before == 2
    torch.cuda.synchronize()
    want = torch.empty_like(y)
    qf.w4a16_linear(_x(M, 1024, torch.bfloat16), ops.SlabWeight(alias.blob.clone(), 128, 1024, 128, torch.bfloat16, target.zero_mode, 8),
                    out=want, out_dtype=torch.float32)
    assert torch.equal(torch.nan_to_num(y), torch.nan_to_num(want))


def test_scales_near_the_top_of_bf16():
    """Scales of 2^126 and more take the converter's other form; K3 has the same one."""
    M, N, K = 9, 256, 256
    sc = _weights(N, K, torch.bfloat16)[1]
    sc[0, ::3] = 2.0 ** 126
    # codes next to the zero point 8, so that every weight is finite
    codes = torch.randint(7, 10, (N, K), dtype=torch.int8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    qw, zr = qf.pack_int4(codes), None
    x = _x(M, K, torch.bfloat16, scale=2.0 ** -126)
    want, got = (torch.empty(M, N, device="cuda") for _ in range(2))
    qf.w4a16_linear(x, qf.prepack_w4(qw), sc, zr, out=want, out_dtype=torch.float32, path=QF_PATH_GEMM,
                    weight_layout=qf.QF_LAYOUT_INTERLEAVED)
    others = [torch.empty_like(got) for _ in range(7)]
    slab = qf.prepack_gemv_slab(qw, sc, zr)
    batch = ops.LinearBatch([(x, slab, out, qf.QF_EPI_NONE, None) for out in [got] + others])
    assert batch.launches() == 1
    batch.run()
    assert bool(want.isfinite().all()) and torch.equal(want, got) and all(torch.equal(want, other) for other in others)


@pytest.mark.parametrize("fuse", [True, False])
def test_stack_runs_as_a_chain(fuse, monkeypatch):
    from quantforge_b200 import stack
    cfg = {"hidden": 4096, "kv": 512, "ffn": 8192, "layers": 2}
    made = []
    for rows in (stack.CHAIN_BATCH, 0):
        monkeypatch.setattr(stack, "CHAIN_BATCH", rows)
        st = stack.DecodeLinearStack(cfg, 11, torch.bfloat16, torch.device("cuda", 0), seed=3, fuse=fuse, epilogues=fuse)
        assert st.chain == (rows > 0)
        st.buf["h_in"].mul_(0.02)
        st.buf["attn"].mul_(0.02)
        st.buf["down"] = torch.empty_like(st.buf["down"])
        st.step()
        st.buf["down"] = torch.empty_like(st.buf["down"])  # a batch made for the old buffer is not used for this one
        st.capture().replay()
        torch.cuda.synchronize()
        made.append({k: v.clone() for k, v in st.buf.items() if k in (("qkv", "o", "act", "down") if fuse else ("q", "k", "v", "o", "gate", "up", "down"))})
    assert all(torch.equal(made[0][k], made[1][k]) for k in made[0])
