"""The linears on host buffers, whichever way the data takes: page-locked buffers that the kernels reach themselves, and, through
the copy engine, larger, pageable and unaligned ones. All give the device call's bits."""
import pytest
import torch

import quantforge_b200 as qf

pytestmark = pytest.mark.gpu


def _layer(N, K, dtype, prepack, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.randn(K // 128, N, device="cuda", generator=gen).abs() * 0.003).clamp_min(2.0 ** -14).to(dtype)
    z = torch.randint(0, 16, (K // 128, N), dtype=torch.int8, device="cuda", generator=gen)
    return qf.W4A16Linear(qw, sc, qf.pack_zeros_u4(z), prepack=prepack)


def _pinned(shape, dtype, offset):
    n = shape[0] * shape[1]
    flat = torch.empty(n + 16, dtype=dtype, pin_memory=True)
    return flat[offset:offset + n].view(shape)


# (1, ...) the GEMV kernel, then narrow and wide tcgen05 tiles; x or y beyond what kernels fetch and write themselves
@pytest.mark.parametrize("M,K,N,prepack", [(1, 512, 512, False), (3, 1024, 256, True), (17, 4096, 1024, True), (200, 1024, 1024, True),
                                           (256, 4096, 512, True), (257, 4096, 512, True), (80, 512, 14336, True)])
@pytest.mark.parametrize("out", ["same", torch.float32])
def test_every_way_gives_the_device_result(M, K, N, prepack, out):
    dtype = torch.bfloat16
    out = dtype if out == "same" else out
    lin = _layer(N, K, dtype, prepack)
    gen = torch.Generator().manual_seed(M)
    x = torch.randn(M, K, generator=gen).to(dtype)
    want = lin(x.cuda(), out_dtype=out).cpu()
    for x_off, y_off, pin_x, pin_y in [(0, 0, True, True), (3, 0, True, True), (0, 5, True, True), (8, 8, True, True),
                                       (0, 0, False, True), (0, 0, True, False)]:
        xh = _pinned((M, K), dtype, x_off) if pin_x else torch.empty(M, K, dtype=dtype)
        yh = _pinned((M, N), out, y_off) if pin_y else torch.empty(M, N, dtype=out)
        xh.copy_(x)
        for wait in (True, False):
            yh.fill_(7)
            lin.forward_host(xh, yh, wait=wait)
            torch.cuda.synchronize()
            assert torch.equal(yh, want)


def test_calls_back_to_back():
    dtype = torch.float16
    a, b = _layer(1024, 512, dtype, True), _layer(512, 512, dtype, True, 1)
    gen = torch.Generator().manual_seed(1)
    xs = [torch.randn(m, 512, generator=gen).to(dtype).pin_memory() for m in (1, 16, 2, 65, 4, 3000) * 3]
    ya = [torch.empty(x.shape[0], 1024, dtype=dtype, pin_memory=True) for x in xs]
    yb = [torch.empty(x.shape[0], 512, dtype=dtype, pin_memory=True) for x in xs]
    for x, m, o in zip(xs, ya, yb):
        a.forward_host(x, m, wait=False)
        b.forward_host(x, o, wait=False)
    torch.cuda.synchronize()
    for x, m, o in zip(xs, ya, yb):
        assert torch.equal(m, a(x.cuda()).cpu())
        assert torch.equal(o, b(x.cuda()).cpu())
