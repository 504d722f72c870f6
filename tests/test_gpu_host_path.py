"""The native host path of the operators (csrc/qf_host.cpp): what it does itself, what it leaves to ops.py, what it raises."""
import ctypes
import json
import os
import shutil
import subprocess
import sys
import threading
import time

import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import _lib, ops
from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu

# The C ABI as the host path calls it, without kernels: counts the calls and returns the status it was told to.
STUB = """
#include <stddef.h>
#include <stdint.h>
int stub_status, stub_calls;
static int call(void) { ++stub_calls; return stub_status; }
const char *qf_status_string(int s) { return "STUB_STATUS"; }
const char *qf_last_error(const void *ctx) { return "stub message"; }
size_t qf_w4a16_workspace_bytes(const void *d) { return 0; }
size_t qf_prepack_bytes(int layout, int64_t N, int64_t K) { return (size_t)(N * K); }
int qf_w4a16_linear_fused() { return call(); }
int qf_unpack_int4() { return call(); }
int qf_pack_int4() { return call(); }
int qf_quantize_w4() { return call(); }
int qf_dequant_w4() { return call(); }
int qf_prepack_gemv_slab() { return call(); }
int qf_prepack_w4() { return call(); }
int qf_prepack_w4_tiled() { return call(); }
"""
CHILD = """
import ctypes, importlib.machinery, importlib.util, json, sys, torch
folder, statuses = sys.argv[1], json.loads(sys.argv[2])
loader = importlib.machinery.ExtensionFileLoader("_qf_host", folder + "/_qf_host.so")
h = importlib.util.module_from_spec(importlib.util.spec_from_loader("_qf_host", loader))
loader.exec_module(h)
stub = ctypes.CDLL(folder + "/libquantforge_rt.so")
status, calls = ctypes.c_int.in_dll(stub, "stub_status"), ctypes.c_int.in_dll(stub, "stub_calls")
class Error(RuntimeError):
    def __init__(self, status, name, message):
        super().__init__(message)
        self.status, self.name = status, name
h.set_error(Error)
h.set_ctx(0, 1)
N, K = 128, 256
dev = "cuda:0"
qw = torch.zeros(N, K // 2, dtype=torch.int8, device=dev)
sc = torch.zeros(K // 128, N, dtype=torch.float16, device=dev)
z = torch.zeros(K // 128, N, dtype=torch.int8, device=dev)
x = torch.zeros(2, K, dtype=torch.float16, device=dev)
out = torch.zeros(2, N, dtype=torch.float16, device=dev)
ops = {
    "linear": lambda: h.linear(x, qw, sc, None, 128, 8, None, 0, 0, None, 0, 0, None),
    "linear into out": lambda: h.linear(x, qw, sc, None, 128, 8, None, 0, 0, out, 0, 0, None),
    "gemv": lambda: h.gemv(x, qw, sc[0], z[0]),
    "unpack": lambda: h.unpack(qw),
    "pack": lambda: h.pack(qw),
    "pack_zeros": lambda: h.pack_zeros(z),
    "quantize": lambda: h.quantize(x, 128, False, torch.float16),
    "dequant": lambda: h.dequant(qw, sc, None, 128, 8),
    "prepack_slab": lambda: h.prepack_slab(qw, sc, None, 128, 8),
    "prepack": lambda: h.prepack(qw, False, 1),
    "prepack tiled": lambda: h.prepack(qw, False, 2),
}
res = {}
for name, fn in ops.items():
    for s in statuses:
        status.value, before = s, calls.value
        try:
            got = "none" if fn() is None else "result"
        except Error as e:
            got = f"{e.status} {e.name} {e}"
        res[f"{name}/{s}"] = [got, calls.value - before]
print(json.dumps(res))
"""


def test_status_of_the_c_call(tmp_path):
    """OK: the result. Refused by the checks in front of the launch: None, ops.py starts over. Anything else may have
    enqueued something: raised, with one call made."""
    (tmp_path / "stub.c").write_text(STUB)
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", str(tmp_path / "libquantforge_rt.so"), str(tmp_path / "stub.c")], check=True)
    shutil.copy(_lib.HOST_PATH, tmp_path / "_qf_host.so")  # it finds the library in its own folder
    refused = [-1, -2, -7]  # QF_ERR_BAD_ARG, QF_ERR_UNSUPPORTED, QF_ERR_WORKSPACE
    raised = [-3, -4, -5, -6]
    assert [_lib.status_name(s) for s in refused] == ["QF_ERR_BAD_ARG", "QF_ERR_UNSUPPORTED", "QF_ERR_WORKSPACE"]
    assert _lib.status_name(-3) == "QF_ERR_CUDA"
    p = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path), json.dumps([0] + refused + raised)], capture_output=True,
                       text=True, env={**os.environ, "LD_LIBRARY_PATH": ""}, timeout=300)
    assert p.returncode == 0, p.stderr
    res = json.loads(p.stdout.strip().splitlines()[-1])
    assert len(res) == 11 * 8
    for key, (got, calls) in res.items():
        s = int(key.rsplit("/", 1)[1])
        want = "result" if s == 0 else "none" if s in refused else f"{s} STUB_STATUS stub message"
        assert (got, calls) == (want, 1), key


def test_an_earlier_error_is_not_the_next_launch_s():
    """A refused allocation inside the library, then operators: one launch each and no error. (out is the residual: a second
    launch would add it twice.)"""
    x = torch.randn(2, 256, device="cuda").half()
    qw = torch.randint(-128, 128, (128, 128), dtype=torch.int8, device="cuda")
    sc = (torch.rand(2, 128, device="cuda") * 0.01).half()
    res = torch.randn(2, 128, device="cuda").half()

    def linear(r):
        return qf.w4a16_linear(x, qw, sc, None, out=r, residual=r, epilogue=qf.QF_EPI_RESIDUAL_ADD)

    calls = {"linear": lambda: linear(res.clone()), "unpack": lambda: qf.unpack_int4(qw), "pack": lambda: qf.pack_int4(qw),
             "dequant": lambda: qf.dequant_w4(qw, sc), "prepack": lambda: qf.prepack_w4(qw),
             "tiled": lambda: qf.prepack_w4(qw, layout=qf.QF_LAYOUT_TILED),
             "slab": lambda: qf.prepack_gemv_slab(qw, sc).blob}
    want = {name: fn() for name, fn in calls.items()}
    for name, fn in calls.items():
        with pytest.raises(qf.QuantForgeError):
            qf.Comm(1 << 42, rank=0, world=1)  # 64 TiB
        before = qf.launch_count()
        got = fn()
        assert qf.launch_count() - before == 1, name
        assert torch.equal(got, want[name]), name


def test_other_threads_run_while_a_launch_blocks():
    """A busy stream and more launches than its queue holds: the launching thread waits in the driver, the others do not."""
    qw = torch.randint(-128, 128, (4, 64), dtype=torch.int8, device="cuda")
    qf.unpack_int4(qw)
    torch.cuda.synchronize()
    longest, stop = 0.0, threading.Event()

    def tick():
        nonlocal longest
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            longest, last = max(longest, now - last), now

    t = threading.Thread(target=tick)
    t.start()
    torch.cuda._sleep(1_000_000_000)  # about half a second
    t0 = time.perf_counter()
    for _ in range(4000):
        qf.unpack_int4(qw)
    blocked = time.perf_counter() - t0
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert blocked > 0.3, "the queue did not fill"
    assert longest < 0.15, (longest, blocked)


def _tensors(act=torch.float16, M=3, N=256, K=512, group=128):
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    t = {"x": torch.randn(M, K, device="cuda", generator=g).to(act), "M": M, "N": N, "K": K, "group": group,
         "qw": torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=g),
         "sc": (torch.rand(K // group, N, device="cuda", generator=g) * 0.01 + 0.001).to(act),
         "z": torch.randint(0, 16, (K // group, N), dtype=torch.int8, device="cuda", generator=g)}
    t["u4"] = qf.pack_zeros_u4(t["z"])
    t["res"] = torch.randn(M, N, device="cuda", generator=g).to(act)
    return t


class Passing(_lib._NoHost):
    """Answers nothing, but hears of contexts and workspaces."""
    set_ctx, add_workspace = staticmethod(_lib.load_host().set_ctx), staticmethod(_lib.load_host().add_workspace)


@pytest.fixture
def python_path(monkeypatch):
    """Runs a call on the Python statements alone."""
    def run(fn):
        with monkeypatch.context() as m:
            m.setattr(ops, "_fast", Passing())
            return fn()
    return run


class Seen:
    """The native host path, noting for each call whether it answered."""

    def __init__(self):
        self.host, self.log = _lib.load_host(), []

    def __getattr__(self, name):
        def call(*args):
            out = getattr(self.host, name)(*args)
            self.log.append((name, out is not None))
            return out
        return call


@pytest.fixture
def seen(monkeypatch):
    s = Seen()
    monkeypatch.setattr(ops, "_fast", s)
    return s


L, I, T = qf.QF_LAYOUT_CANONICAL, qf.QF_LAYOUT_INTERLEAVED, qf.QF_LAYOUT_TILED
ORDINARY = {
    "canonical u4": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"]),
    "canonical i8": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["z"]),
    "canonical const": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], None, zero_const=7),
    "uint8 weights": lambda t: qf.w4a16_linear(t["x"], t["qw"].view(torch.uint8), t["sc"], t["u4"]),
    "int32 weights": lambda t: qf.w4a16_linear(t["x"], t["qw"].view(torch.int32), t["sc"], t["u4"]),
    "fp32 out": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], out_dtype=torch.float32),
    "split": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], split_k=2),
    "residual": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], residual=t["res"], epilogue=qf.QF_EPI_RESIDUAL_ADD),
    "silu": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], epilogue=qf.QF_EPI_SILU_MUL),
    "slab": lambda t: qf.w4a16_linear(t["x"], qf.prepack_gemv_slab(t["qw"], t["sc"], t["u4"])),
    "layer": lambda t: qf.W4A16Linear(t["qw"], t["sc"], t["u4"], prepack=True)(t["x"]),
    "parameter": lambda t: qf.w4a16_linear(torch.nn.Parameter(t["x"]), t["qw"], t["sc"], t["u4"]),
    "gemv": lambda t: qf.gemv_int4(t["x"], t["qw"], t["sc"][0].contiguous(), t["z"][0].contiguous()),
    "unpack": lambda t: qf.unpack_int4(t["qw"]),
    "unpack 3d": lambda t: qf.unpack_int4(t["qw"].view(2, -1, t["K"] // 2)),
    "pack": lambda t: qf.pack_int4(t["z"]),
    "pack_zeros": lambda t: qf.pack_zeros_u4(t["z"]),
    "quantize": lambda t: torch.cat([a.float().flatten() for a in quantize_w4(t["x"], 128)]),
    "dequant": lambda t: qf.dequant_w4(t["qw"], t["sc"], t["u4"]),
    "prepack": lambda t: qf.prepack_w4(t["qw"]),
    "prepack tiled": lambda t: qf.prepack_w4(t["qw"], layout=T),
    "prepack back": lambda t: qf.prepack_w4(t["qw"], to_canonical=True, layout=T),
    "prepack slab": lambda t: qf.prepack_gemv_slab(t["qw"], t["sc"], t["z"]).blob,
}
# answered by ops.py: a copy to make, or a form that only it reads
PASSED_ON = {
    "x not contiguous": lambda t: qf.w4a16_linear(t["x"].t().contiguous().t(), t["qw"], t["sc"], t["u4"]),
    "weights not contiguous": lambda t: qf.w4a16_linear(t["x"], t["qw"].t().contiguous().t(), t["sc"], t["u4"]),
    "scales not contiguous": lambda t: qf.dequant_w4(t["qw"], t["sc"].t().contiguous().t(), t["u4"]),
    "gemv, zero points of uint8": lambda t: qf.gemv_int4(t["x"], t["qw"], t["sc"][0].contiguous(), t["z"][0].view(torch.uint8)),
    "no rows": lambda t: qf.w4a16_linear(t["x"][:0], t["qw"], t["sc"], t["u4"]),
    "zero_const as a float": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], None, zero_const=8.0),
    "codes not contiguous": lambda t: qf.pack_int4(t["z"].t().contiguous().t()),
    "codes not aligned": lambda t: qf.pack_int4(t["z"].flatten()[1:-1]),
    "quantise to fp32 scales": lambda t: quantize_w4(t["x"], 128, True, torch.float32)[1],
    "quantise odd groups": lambda t: quantize_w4(t["x"][:, :510], 510)[1],
    "nothing to unpack": lambda t: qf.unpack_int4(t["qw"][:0]),
}
REFUSED = {
    "x of another type": lambda t: qf.w4a16_linear(t["x"].float(), t["qw"], t["sc"], t["u4"]),
    "x too short": lambda t: qf.w4a16_linear(t["x"][:, :256].contiguous(), t["qw"], t["sc"], t["u4"]),
    "x of three dimensions": lambda t: qf.w4a16_linear(t["x"][None], t["qw"], t["sc"], t["u4"]),
    "x misaligned": lambda t: qf.w4a16_linear(torch.cat([t["x"].flatten()] * 2)[1:1 + t["x"].numel()].view(t["x"].shape), t["qw"], t["sc"], t["u4"]),
    "x on the CPU": lambda t: qf.w4a16_linear(t["x"].cpu(), t["qw"], t["sc"], t["u4"]),
    "zeros of another shape": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["z"][:1].contiguous()),
    "zeros of another type": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["z"].short()),
    "group of 0": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], group_size=0),
    "residual missing": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], epilogue=qf.QF_EPI_RESIDUAL_ADD),
    "residual of another type": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], residual=t["res"].float(),
                                                          epilogue=qf.QF_EPI_RESIDUAL_ADD),
    "out of another shape": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], out=t["res"][:1]),
    "zero_const out of range": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], None, zero_const=300),
    "layout unknown": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], weight_layout=9),
    "negative split": lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], split_k=-1),
    "slab of too many rows": lambda t: qf.w4a16_linear(t["x"].repeat(20, 1), qf.prepack_gemv_slab(t["qw"], t["sc"], t["u4"])),
    "unpack floats": lambda t: qf.unpack_int4(t["x"]),
    "pack floats": lambda t: qf.pack_int4(t["x"]),
}


@pytest.mark.parametrize("act", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("name", list(ORDINARY))
def test_ordinary_calls_are_answered_natively_and_alike(seen, python_path, name, act):
    t = _tensors(act)
    want = python_path(lambda: ORDINARY[name](t))  # also makes context and workspace
    seen.log.clear()
    got = ORDINARY[name](t)
    assert seen.log and all(ok for _, ok in seen.log), seen.log
    assert got.dtype == want.dtype and torch.equal(got, want)


@pytest.mark.parametrize("name", list(PASSED_ON))
def test_other_calls_are_passed_on(seen, python_path, name):
    t = _tensors()
    want = python_path(lambda: PASSED_ON[name](t))
    seen.log.clear()
    got = PASSED_ON[name](t)
    assert any(not ok for _, ok in seen.log), seen.log
    assert got.shape == want.shape and torch.equal(got, want)


@pytest.mark.parametrize("name", list(REFUSED))
def test_calls_in_error_are_refused_alike(python_path, name):
    t = _tensors()
    qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"])
    errors = []
    for run in (lambda fn: fn(), python_path):
        with pytest.raises(Exception) as e:
            run(lambda: REFUSED[name](t))
        errors.append((type(e.value), str(e.value)))
    assert errors[0] == errors[1]


def test_results_go_where_the_caller_says(python_path):
    t = _tensors()
    want = python_path(lambda: ORDINARY["residual"](t))
    y = t["res"].clone()  # out is the residual
    got = qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], residual=y, out=y, epilogue=qf.QF_EPI_RESIDUAL_ADD)
    assert got is y and torch.equal(y, want)


def test_streams_and_growing_workspaces(seen, python_path):
    """A stream's first call that needs scratch is passed on and makes it; later ones that fit are answered natively. Results on
    two streams at once are those of one."""
    small, large = _tensors(M=16, N=1024, K=4096), _tensors(M=64, N=8192, K=4096)
    call = lambda t: qf.w4a16_linear(t["x"], t["qw"], t["sc"], t["u4"], split_k=16)  # noqa: E731
    want = [python_path(lambda t=t: call(t)) for t in (small, large)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for s in streams:
        with torch.cuda.stream(s):
            for t in (small, small, large, large, small):
                seen.log.clear()
                call(t)
    got = []
    for i in range(6):
        for s in streams:
            with torch.cuda.stream(s):
                seen.log.clear()
                got.append((i % 2, call((small, large)[i % 2])))
                assert seen.log == [("linear", True)]
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[k]) for k, y in got)
    # a stream of its own: torch hands out those of its pool in turn, and any of them may have a workspace from an earlier test
    handle = ctypes.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(handle))) == 0
    assert (torch.cuda.current_device(), handle.value) not in ops._workspaces
    fresh = torch.cuda.ExternalStream(handle.value)
    with torch.cuda.stream(fresh):
        answered = []
        for t in (small, small, large, large, small):
            seen.log.clear()
            call(t)
            answered.append(seen.log[0][1])
    assert answered[0] is False and answered[1] is True and answered[3] is True and answered[4] is True
    torch.cuda.synchronize()
