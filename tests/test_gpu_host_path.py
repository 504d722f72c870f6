"""The native host path of the operators (csrc/qf_host.cpp): what it does itself, what it leaves to ops.py, what it raises."""
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
from quantforge_b200 import _lib

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
