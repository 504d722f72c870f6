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
@pytest.mark.parametrize("group", [128, 64, 512])
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
