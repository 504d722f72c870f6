"""Quotients by the reciprocal and its residual in the quantise kernels: the codes and zero points of divisions, bit for bit, at ties, for
scales of all sizes, next to where the kernels divide instead, and for values that are nothing beside the scale."""
import pytest
import torch

from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu


def _same(w, group, symmetric, scale_dtype=None):
    got = quantize_w4(w, group, symmetric, scale_dtype)
    want = quantize_w4(w.clone().requires_grad_(), group, symmetric, scale_dtype)  # autograd watches: the tensor program
    for a, b in zip(got, want):
        if a is not None:
            b = b.detach()
            assert a.dtype == b.dtype and torch.equal(torch.nan_to_num(a.float(), nan=-1.0), torch.nan_to_num(b.float(), nan=-1.0))


@pytest.mark.parametrize("dtype,scale_dtype", [(torch.float16, None), (torch.bfloat16, None), (torch.float32, torch.bfloat16), (torch.float32, torch.float16)])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("group", [128, 64, 256, 512, 1024, 640])
def test_quotients(dtype, scale_dtype, symmetric, group):
    gen = torch.Generator(device="cuda").manual_seed(group)
    rnd = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)  # noqa: E731
    half = dtype == torch.float16 or scale_dtype == torch.float16
    rows = [rnd(2048, group) * 0.02]                                          # ties as they come: one in 500 of bf16 weights
    k = torch.randint(-8, 8, (1024, group), device="cuda", generator=gen).float() + 0.5
    scale = (rnd(1024, 1).abs() + 0.01).to(torch.float16 if half else torch.bfloat16).float()
    rows.append(k * scale)                                                    # halves of a 16-bit scale, on and next to the ties
    rows.append(k * scale + scale * 2.0 ** -9 * rnd(1024, group).sign())
    exponents = torch.linspace(-20, 12 if half else 121, 512, device="cuda").round()[:, None]
    rows.append(rnd(512, group) * 2.0 ** exponents)                           # scales up to the largest, 2^-14 at least
    rows.append((rnd(512, group) * 1e-3 + 2.0 ** torch.linspace(-3, 10, 512, device="cuda")[:, None]))  # quotients around 256 and above
    tiny = rnd(64, group) * 2.0 ** torch.randint(-149 if not half else -24, 0, (64, group), device="cuda", generator=gen).float()
    tiny[:, 0] = 7.0
    rows.append(tiny)
    _same(torch.cat(rows).to(dtype), group, symmetric, scale_dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("N,K,group", [(3, 768, 256), (17, 1024, 512), (33, 512, 256), (5, 1040, 1040), (2, 4096, 1024), (3, 2064, 2064), (2, 4096, 4096),
                                       (2, 8192, 4096), (3, 4112, 4112), (1, 8192, 8192), (2, 8208, 8208), (2, 28672, 28672), (70000, 512, 512), (1, 20, 20)])
def test_large_groups(N, K, group, dtype, symmetric):
    gen = torch.Generator(device="cuda").manual_seed(K)
    w = (torch.randn(N, K, device="cuda", generator=gen) * 0.05).to(dtype)
    _same(w, group, symmetric)
    if N < 100:  # extremes and NaN at the ends of what a thread, a tile and a group hold
        for i, at in enumerate((0, group - 1, group // 2, min(group - 1, 15), min(group - 1, 4095), min(group - 1, 8191))):
            v = w.clone()
            v[i % N, at], v[i % N, (at + 7) % group] = 3.0, -2.0
            _same(v, group, symmetric)
            v[i % N, at] = float("nan")
            _same(v, group, symmetric)
