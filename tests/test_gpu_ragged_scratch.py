"""Canonical weights of a ragged row count with the scratch of the GEMV kernel only, or none: that kernel serves the call, as it did
before the tcgen05 kernel took such weights; with less the call is refused."""
import ctypes

import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200 import _lib, ops

pytestmark = pytest.mark.gpu


# splits of the GEMV kernel: 12 (through memory), 5 (on chip), none, none, 2, none (as the tcgen05 kernel)
@pytest.mark.parametrize("M,K,N", [(8, 6144, 1040), (16, 8192, 4112), (64, 4096, 4112), (200, 4096, 4112), (300, 8192, 1040), (300, 512, 28688)])
def test_scratch_of_the_gemv_kernel(M, K, N):
    lib, dev = _lib.load(), torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device="cuda").manual_seed(K + N)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device=dev, generator=gen)
    sc = (torch.rand(K // 128, N, device=dev, generator=gen) * 0.003 + 0.0005).bfloat16()
    x = torch.randn(M, K, device=dev, generator=gen).bfloat16()

    def desc(path):
        return _lib.LinearDesc(M=M, N=N, K=K, group_size=128, act_dtype=_lib.QF_BF16, out_dtype=_lib.QF_BF16, zero_mode=_lib.QF_ZERO_CONST,
                               zero_const=8, path=path)

    def call(d, scratch):
        y = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=dev)
        ws = torch.zeros(scratch, dtype=torch.uint8, device=dev) if scratch else None
        ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
        st = lib.qf_w4a16_linear(ops._ctx(dev), ctypes.byref(d), ptr(x), ptr(qw), ptr(sc), None, ptr(y), ptr(ws), scratch,
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        return st, y

    auto, gemv = desc(_lib.QF_PATH_AUTO), desc(_lib.QF_PATH_GEMV)
    own, both = (int(lib.qf_w4a16_workspace_bytes(ctypes.byref(d))) for d in (gemv, auto))
    assert own < both or both == 0
    st, want = call(gemv, own)
    assert st == 0
    st, y = call(auto, own)
    # where neither kernel splits there is no reason to leave the faster one, whose order of sums shows in some roundings
    assert st == 0 and torch.equal(y, want) == (own < both)
    st, y = call(auto, both)
    # both round sums of at most 1e-4 of the outputs' rms apart to bf16
    e = 1e-4 * float(want.float().pow(2).mean().sqrt())
    assert st == 0 and bool(((y.float() - want.float()).abs() <= e + 2.0 ** -7 * (want.float().abs() + e)).all())
    if own:
        st, y = call(auto, own - 16)
        assert st == -7 and bool((y == 7.0).all())  # QF_ERR_WORKSPACE
    assert qf.device_status() == 0
