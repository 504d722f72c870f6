"""What the linears on host buffers promise beside the result: nothing enqueued by a call that is refused, and order between calls
of several streams, threads and buffers."""
import ctypes
import threading

import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _layer(N, K, dtype=torch.float16, prepack=False, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // 128, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    z = torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen)
    return qf.W4A16Linear(qw, sc, qf.pack_zeros_u4(z), prepack=prepack)


def _c_call(d, x, qw, sc, z, y, ws, ws_bytes):
    lib, ctx = _lib.load(), ops._ctx(qw.device)
    st = lib.qf_w4a16_linear_host_async(ctx, ctypes.byref(d), x.data_ptr(), qw.data_ptr(), sc.data_ptr(), z.data_ptr(), y.data_ptr(),
                                        ws.data_ptr() if ws is not None else 0, ws_bytes, torch.cuda.current_stream().cuda_stream)
    return _lib.status_name(st)


@pytest.mark.parametrize("pinned", [True, False])
def test_a_refused_call_enqueues_nothing(pinned):
    lin = _layer(4096, 4096)
    x, y = torch.randn(2, 4096).half(), torch.zeros(2, 4096, dtype=torch.float16)
    if pinned:
        x, y = x.pin_memory(), y.pin_memory()
    lin.forward_host(x, y)
    torch.cuda.synchronize()
    y.zero_()

    def desc(M=2, N=4096, K=4096):
        return ops._make_desc(M, N, K, 128, torch.float16, torch.float16, lin.zeros, 8, 0, 0)

    need = qf.workspace_bytes(desc())
    assert need > 0
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    args = (x, lin.qweight, lin.scales, lin.zeros, y)
    before = qf.launch_count()
    assert _c_call(desc(), *args, ws, need - 1) == "QF_ERR_WORKSPACE"
    assert _c_call(desc(), *args, None, 0) == "QF_ERR_WORKSPACE"
    assert _c_call(desc(M=1, K=4), *args, ws, need) == "QF_ERR_BAD_ARG"  # eight bytes of activations
    assert _c_call(desc(K=4096 - 64), *args, ws, need) == "QF_ERR_BAD_ARG"
    d = desc()
    d.epilogue = _lib.QF_EPI_RESIDUAL_ADD
    assert _c_call(d, *args, ws, need) == "QF_ERR_BAD_ARG"
    d = desc()
    d.reserved[0] = 1
    assert _c_call(d, *args, ws, need) == "QF_ERR_BAD_ARG"
    torch.cuda.synchronize()
    assert qf.launch_count() == before and not y.any()
    assert _c_call(desc(), *args, ws, need) == "QF_OK"
    torch.cuda.synchronize()
    assert torch.equal(y, lin(x.cuda()).cpu())


@pytest.mark.parametrize("pinned", [True, False])
def test_a_capture_refuses_and_goes_on(pinned):
    """Host buffers are not part of a graph; the call says so and leaves the capture as it was."""
    lin = _layer(512, 512)
    x, y = torch.randn(2, 512).half(), torch.zeros(2, 512, dtype=torch.float16)
    if pinned:
        x, y = x.pin_memory(), y.pin_memory()
    xd = x.cuda()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        lin.forward_host(x, y)
        lin(xd)
    want = y.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        with pytest.raises(_lib.QuantForgeError):
            lin.forward_host(x, y, wait=False)
        out = lin(xd)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want)


def test_each_stream_has_its_own_workspace(monkeypatch):
    """A layer that was called on one stream and then on another passes each call the scratch of the stream it runs on: split sums
    of device calls on the first stream may be under way."""
    lin = _layer(4096, 4096)
    x, y = torch.randn(2, 4096).half().pin_memory(), torch.empty(2, 4096, dtype=torch.float16, pin_memory=True)
    real, passed = _lib.load().qf_w4a16_linear_host, []

    class Lib:
        def __getattr__(self, name):
            return getattr(_LIB, name)

        def qf_w4a16_linear_host(self, *args):
            passed.append((args[-1], args[7].value))
            return real(*args)

    _LIB = _lib.load()
    monkeypatch.setattr(_lib, "load", Lib)
    streams = [torch.cuda.Stream() for _ in range(3)]
    for s in streams * 2:
        with torch.cuda.stream(s):
            lin.forward_host(x, y)
    assert len({stream for stream, _ in passed}) == 3 and len({ws for _, ws in passed}) == 3
    for stream, ws in passed:
        assert ws in {b.data_ptr() for b in ops._workspaces[(0, stream)]}


def test_activations_of_another_width_are_refused():
    lin = _layer(512, 512)
    y = torch.empty(2, 512, dtype=torch.float16, pin_memory=True)
    lin.forward_host(torch.randn(2, 512).half().pin_memory(), y)
    with pytest.raises(ValueError):
        lin.forward_host(torch.randn(2, 256).half().pin_memory(), y)


def _calls(lin, K, N, rows, pinned, seed):
    """(activations, result, device call's result) of calls on `lin`, one per entry of `rows`."""
    gen = torch.Generator().manual_seed(seed)
    out = []
    for m in rows:
        x, y = torch.randn(m, K, generator=gen).half(), torch.empty(m, N, dtype=torch.float16)
        out.append((x.pin_memory(), y.pin_memory()) if pinned else (x, y))
    want = [lin(x.cuda()).cpu() for x, _ in out]
    torch.cuda.synchronize()
    return [(x, y, w) for (x, y), w in zip(out, want)]


# few rows: fetched by a kernel; 1100 rows of 1024: copied; a mixture of both
ROWS = {"fetched": [2, 16, 1, 64, 33, 5], "copied": [1100, 1300, 1024 + 9], "mixed": [2, 1100, 64, 1100, 7, 40]}


@pytest.mark.parametrize("kind", sorted(ROWS))
@pytest.mark.parametrize("order", ["abab", "aabb", "abbaab"])
def test_streams_side_by_side(kind, order):
    """One thread, two streams, a layer for each, no wait between the calls: everybody gets its own rows."""
    K = N = 1024
    lins = {c: _layer(N, K, prepack=True, seed=i) for i, c in enumerate("ab")}
    streams = {c: torch.cuda.Stream() for c in "ab"}
    calls = {c: _calls(lins[c], K, N, ROWS[kind] * 4, True, i) for i, c in enumerate("ab")}
    todo = {c: list(calls[c]) for c in "ab"}
    while todo["a"] or todo["b"]:
        for c in order:
            if todo[c]:
                x, y, _ = todo[c].pop(0)
                with torch.cuda.stream(streams[c]):
                    lins[c].forward_host(x, y, wait=False)
    torch.cuda.synchronize()
    for c in "ab":
        for _, y, want in calls[c]:
            assert torch.equal(y, want)


@pytest.mark.parametrize("kind", sorted(ROWS))
@pytest.mark.parametrize("wait", [True, False])
@pytest.mark.parametrize("own_streams", [False, True])
def test_threads_side_by_side(kind, wait, own_streams):
    """Four threads with a layer each, on streams of their own or all on the same one."""
    K = N = 1024
    lins = [_layer(N, K, prepack=True, seed=i) for i in range(4)]
    calls = [_calls(lin, K, N, ROWS[kind] * 6, True, i) for i, lin in enumerate(lins)]
    start, errors = threading.Barrier(4), []

    def work(i):
        try:
            start.wait()
            with torch.cuda.stream(torch.cuda.Stream() if own_streams else torch.cuda.default_stream()):
                for x, y, _ in calls[i]:
                    lins[i].forward_host(x, y, wait=wait)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for per_layer in calls:
        for _, y, want in per_layer:
            assert torch.equal(y, want)


def test_one_staging_for_each_stream():
    """Calls on two streams go through contexts of their own, found again by the next call on the stream."""
    lin = _layer(512, 512)
    x, y = torch.randn(2, 512).half().pin_memory(), torch.empty(2, 512, dtype=torch.float16, pin_memory=True)
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in streams * 2:
        with torch.cuda.stream(s):
            lin.forward_host(x, y)
            qf.w4a16_linear_host(x, lin.qweight, lin.scales, lin.zeros, out_host=y)
    ctxs = [ops._host_ctxs[(0, s.cuda_stream)].value for s in streams]
    assert len(set(ctxs)) == 2 and ops._ctx(lin.qweight.device).value not in ctxs
    assert {prep[2].value for prep in lin._host_prep.values()} == set(ctxs)
    assert qf.device_status() == 0


# rows of the chain's layers; "mixed": the second layer takes a part of what the first one wrote
@pytest.mark.parametrize("rows", [(4, 4, 4), (64, 64, 64), (1100, 1100, 1100), (1100, 1000, 17), (40, 1100, 1100)])
@pytest.mark.parametrize("in_front", [False, True])
def test_the_result_of_one_call_is_the_activations_of_the_next(rows, in_front):
    """Without a wait in between, page-locked: fetched, copied, and from one to the other. Behind work that keeps the GPU busy, and
    with more results pending than the context keeps a list of."""
    K = N = 1024
    lins = [_layer(N, K, prepack=True, seed=i) for i in range(3)]
    big = max(rows)
    busy = _layer(8192, 8192, prepack=True, seed=9)
    gen = torch.Generator().manual_seed(sum(rows))
    runs = []
    for _ in range(7):
        bufs = [torch.zeros(big, N, dtype=torch.float16, pin_memory=True) for _ in range(4)]
        bufs[0].copy_(torch.randn(big, K, generator=gen))
        want = [bufs[0].clone()] + [b.clone() for b in bufs[1:]]
        for i, m in enumerate(rows):
            want[i + 1][:m] = lins[i](want[i][:m].cuda()).cpu()
        runs.append((bufs, want))
    xb = torch.randn(256, 8192, device="cuda").half()
    torch.cuda.synchronize()
    for _ in range(3):
        for bufs, _ in runs:
            for b in bufs[1:]:
                b.zero_()
        for bufs, _ in runs:
            if in_front:
                busy(xb)
            for i, m in enumerate(rows):
                lins[i].forward_host(bufs[i][:m], bufs[i + 1][:m], wait=False)
        torch.cuda.synchronize()
        for bufs, want in runs:
            for i, m in enumerate(rows):
                assert torch.equal(bufs[i + 1][:m], want[i + 1][:m])


# M, K, N, tiled weights, fp32 result, way: page-locked and aligned
WAYS = [(1, 512, 512, False, False, "fetched"), (2, 4096, 4096, False, True, "fetched"), (64, 512, 512, True, False, "fetched"),
        (256, 4096, 4096, True, False, "fetched"), (257, 4096, 4096, True, False, "copied"), (80, 512, 14336, True, False, "copied"),
        (64, 4096, 8192, True, True, "fetched"), (64, 4096, 8192 + 128, True, True, "copied"),
        # fp32 from the tcgen05 kernel: without a split up to 192 KB
        (96, 512, 512, True, True, "fetched"), (97, 512, 512, True, True, "copied"), (1000, 512, 512, True, True, "copied"),
        (1000, 512, 512, True, False, "fetched"), (256, 4096, 2048, True, True, "fetched")]


@pytest.mark.parametrize("M,K,N,prepack,wide,way", WAYS)
def test_which_way(M, K, N, prepack, wide, way):
    """A fetched call is one launch more than a copied one; pageable and unaligned buffers are copied whatever their size."""
    lin = _layer(N, K, prepack=prepack)
    out = torch.float32 if wide else torch.float16
    x = torch.randn(M * K + 8).half()
    want = lin(x[:M * K].view(M, K).cuda(), out_dtype=out).cpu()
    xp, yp = x.pin_memory(), torch.empty(M * N + 8, dtype=out, pin_memory=True)
    xu = torch.empty(M * K + 8, dtype=torch.float16, pin_memory=True)
    xu[1:1 + M * K] = x[:M * K]
    y = yp[:M * N].view(M, N)
    lin.forward_host(xp[:M * K].view(M, K), y)
    for xh, yh, expected in [(xp[:M * K], yp[:M * N], way), (x[:M * K], yp[:M * N], "copied"), (xp[:M * K], torch.empty(M * N, dtype=out), "copied"),
                             (xu[1:1 + M * K], yp[:M * N], "copied"), (xp[:M * K], yp[1:1 + M * N], "copied")]:
        before = qf.launch_count()
        lin.forward_host(xh.view(M, K), yh.view(M, N))
        assert qf.launch_count() - before == (2 if expected == "fetched" else 1)
        assert torch.equal(yh.view(M, N), want)
