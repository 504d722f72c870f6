"""The layout helpers under what watches tensor programs: autograd, forward mode, tracers, function transforms, subclasses."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu


def _w(seed, N=8, K=256):
    return torch.randn(N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)) * 0.1


def _codes(seed, shape=(8, 64)):
    return torch.randint(0, 16, shape, dtype=torch.int8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


HELPERS = {"pack": (qf.pack_int4, _codes), "pack_zeros": (qf.pack_zeros_u4, _codes),
           "quantise": (lambda w: quantize_w4(w, 128), _w), "quantise symmetric": (lambda w: quantize_w4(w, 128, True)[:2], _w)}


def _same(a, b):
    a, b = [t if isinstance(t, (tuple, list)) else (t,) for t in (a, b)]
    return len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("layer", [True, False])
def test_quantise_gives_scales_their_gradient(symmetric, layer):
    w = _w(0)
    leaf = torch.nn.Parameter(w) if layer else w.clone().requires_grad_()
    scales = quantize_w4(leaf, 128, symmetric, torch.float16)[1]
    assert scales.requires_grad
    scales.float().sum().backward()
    want = w.cpu().requires_grad_()  # amax and amin pass their gradient to the extreme elements: no rounding but 1/15 or 1/7
    quantize_w4(want, 128, symmetric, torch.float16)[1].float().sum().backward()
    assert torch.allclose(leaf.grad.cpu(), want.grad, rtol=1e-6, atol=0)
    with torch.no_grad():
        before = qf.launch_count()
        assert torch.equal(quantize_w4(leaf, 128, symmetric, torch.float16)[1], scales)
        assert qf.launch_count() == before + 1


def test_quantise_forward_mode():
    import torch.autograd.forward_ad as fwad
    with fwad.dual_level():
        scales = quantize_w4(fwad.make_dual(_w(0), torch.ones_like(_w(0))), 128, True)[1]
        assert fwad.unpack_dual(scales).tangent is not None


@pytest.mark.parametrize("name", list(HELPERS))
def test_make_fx_records_the_program(name):
    from torch.fx.experimental.proxy_tensor import make_fx
    fn, make = HELPERS[name]
    fn(make(0))
    g = make_fx(fn)(make(1))
    assert _same(g(make(2)), fn(make(2)))


@pytest.mark.parametrize("name", list(HELPERS))
def test_compiled_in_one_graph(name):
    fn, make = HELPERS[name]
    fn(make(0))
    c = torch.compile(fn, fullgraph=True, backend="eager")
    assert _same(c(make(1)), fn(make(1)))


@pytest.mark.parametrize("name", ["pack", "pack_zeros", "quantise symmetric"])
def test_jit_trace(name):
    fn, make = HELPERS[name]
    fn(make(0))
    g = torch.jit.trace(fn, (make(1),), check_trace=False)
    assert _same(g(make(2)), fn(make(2)))


def test_vmap_over_packing():
    codes = _codes(0, (3, 8, 64))
    qf.pack_int4(codes)
    assert torch.equal(torch.vmap(qf.pack_int4)(codes), torch.stack([qf.pack_int4(c) for c in codes]))


def test_subclasses_and_modes_see_the_operators():
    from torch.utils._python_dispatch import TorchDispatchMode

    class Logged(torch.Tensor):
        pass

    class Count(TorchDispatchMode):
        n = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.n += 1
            return func(*args, **(kwargs or {}))

    codes = _codes(0)
    want = qf.pack_int4(codes)
    got = qf.pack_int4(codes.as_subclass(Logged))
    assert type(got) is Logged and torch.equal(got.as_subclass(torch.Tensor), want)
    with Count() as mode:
        assert torch.equal(qf.pack_int4(codes), want)
    assert mode.n > 2


def test_first_call_of_a_process_inside_a_capture():
    """Without a context yet the helpers are recorded as tensor programs."""
    import subprocess
    import sys
    code = """
import torch
import quantforge_b200 as qf
from quantforge_b200.quantize import quantize_w4
codes = torch.randint(0, 16, (8, 64), dtype=torch.int8, device="cuda")
w = torch.randn(8, 256, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    got = [qf.pack_int4(codes), qf.pack_zeros_u4(codes), *quantize_w4(w, 128)]
codes.copy_(15 - codes)
w.neg_()
g.replay()
torch.cuda.synchronize()
assert qf.launch_count() == 0
want = [qf.pack_int4(codes), qf.pack_zeros_u4(codes), *quantize_w4(w, 128)]
assert qf.launch_count() == 3
assert all(torch.equal(a, b) for a, b in zip(got, want))
"""
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
