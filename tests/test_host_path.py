"""The native host path is for one interpreter and one torch; the package works without it."""
import subprocess
import sys
import sysconfig
import warnings

import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import _lib, build, ops


def test_named_after_interpreter_and_torch():
    assert sysconfig.get_config_var("SOABI") in _lib.HOST_PATH and torch.__version__ in _lib.HOST_PATH
    assert build.build_host() == _lib.HOST_PATH


def test_a_copy_for_another_torch_is_not_up_to_date(monkeypatch, tmp_path):
    other = tmp_path / "_qf_host.other.so"
    monkeypatch.setattr(_lib, "HOST_PATH", str(other))
    commands = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: commands.append(cmd))
    assert build.build_host() == str(other)
    assert len(commands) == 1 and str(other) in commands[0]


@pytest.mark.parametrize("content", [None, b"not a library"])
def test_operators_without_it(monkeypatch, tmp_path, content):
    path = tmp_path / "_qf_host.so"
    if content is not None:
        path.write_bytes(content)
    monkeypatch.setattr(_lib, "HOST_PATH", str(path))
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(ops, "_fast", None)
    with pytest.warns(RuntimeWarning, match="native host path"):
        with pytest.raises(ValueError, match="CUDA tensors only"):  # what the Python statements say to a CPU tensor
            qf.unpack_int4(torch.zeros(4, 4, dtype=torch.int8))
    with warnings.catch_warnings():
        warnings.simplefilter("error")  # said once
        with pytest.raises(ValueError, match="CUDA tensors only"):
            qf.dequant_w4(torch.zeros(16, 64, dtype=torch.int8), torch.zeros(1, 16).half())


@pytest.mark.gpu
def test_operators_on_a_gpu_with_and_without_it():
    """A child process without any built library packs and quantises CUDA tensors as tensor programs, and says what is missing
    where only the library can answer; one without the host path alone computes the same bits as with it."""
    code = """
import sys, warnings
warnings.simplefilter("ignore")
import torch
from quantforge_b200 import _lib
which = sys.argv[1]
if which != "all":
    _lib.HOST_PATH += ".missing"
if which == "none":
    _lib.LIB_PATH += ".missing"
import quantforge_b200 as qf
from quantforge_b200.quantize import quantize_w4
g = torch.Generator(device="cuda").manual_seed(0)
w = torch.randn(128, 256, device="cuda", generator=g).half()
codes, scales, zeros = quantize_w4(w, 128)
qw, qz = qf.pack_int4(codes), qf.pack_zeros_u4(zeros)
x = torch.randn(2, 256, device="cuda", generator=g).half()
try:
    y = [qf.w4a16_linear(x, qw, scales, qz), qf.dequant_w4(qw, scales, qz), qf.unpack_int4(qw),
         qf.w4a16_linear(x, qf.prepack_gemv_slab(qw, scales, qz)), qf.prepack_w4(qw, layout=qf.QF_LAYOUT_TILED)]
except ImportError as e:
    assert which == "none" and "is missing: build it" in str(e)
    y = []
print([int(t.view(torch.uint8).long().mul(torch.arange(t.view(torch.uint8).numel(), device="cuda").view(t.view(torch.uint8).shape) % 251 + 1).sum())
       for t in [qw, qz, scales, *y]])
"""
    out = {}
    for which in ("all", "rt", "none"):
        p = subprocess.run([sys.executable, "-c", code, which], capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr
        out[which] = eval(p.stdout.strip().splitlines()[-1])
    assert out["all"] == out["rt"]
    assert out["none"] == out["all"][:3]
