"""The group-of-128 quantise kernel against the tensor statement on CUDA, bit for bit, where its packed arithmetic could differ:
row counts around a block's 16, quotients at and next to the rounding boundaries, infinities, NaN and signed zeros."""
import pytest
import torch

from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu


def _same(w, symmetric):
    got = quantize_w4(w, 128, symmetric)
    want = quantize_w4(w.clone().requires_grad_(), 128, symmetric)  # autograd watches: the tensor program
    for a, b in zip(got, want):
        if a is None:
            assert b is None
            continue
        b = b.detach()
        assert a.dtype == b.dtype and a.shape == b.shape
        if a.is_floating_point():
            a, b = torch.nan_to_num(a.float(), nan=-1.0), torch.nan_to_num(b.float(), nan=-1.0)
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("N,K", [(1, 128), (15, 640), (16, 512), (17, 384), (33, 128)])
def test_row_counts(N, K, dtype, symmetric):
    gen = torch.Generator(device="cuda").manual_seed(N)
    _same((torch.randn(N, K, device="cuda", generator=gen) * 0.05).to(dtype), symmetric)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("symmetric", [False, True])
def test_rounding_boundaries(dtype, symmetric):
    # ranges of 15 (or +-7) powers of two make the scale a power of two, so that halves are ties; steps of 2^-6 around them
    steps = torch.arange(128, device="cuda", dtype=torch.float32)
    rows = []
    for scale in (2.0 ** -9, 2.0 ** -6, 0.25, 3.0):
        for shift in (-7.0, -7.5, 0.0, -15.0, 4.0):
            base = (steps % 15) + shift + ((steps // 15) - 4) * 0.5 * 2.0 ** -6 + 0.5
            base = base.clamp(shift, shift + 15)
            base[0], base[1] = shift, shift + 15
            rows.append(base * scale)
    _same(torch.stack(rows).to(dtype), symmetric)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("symmetric", [False, True])
def test_special_values(dtype, symmetric):
    inf, nan = float("inf"), float("nan")
    gen = torch.Generator(device="cuda").manual_seed(3)
    w = torch.randn(12, 128, device="cuda", generator=gen) * 0.1
    w[0] = 0.0
    w[1] = -0.0
    w[2] = 1000.0
    w[3] = -1000.0
    w[4] = torch.linspace(99.0, 100.0, 128, device="cuda")    # zero point far below the range
    w[5] = torch.linspace(-100.0, -99.0, 128, device="cuda")  # and far above
    w[6] = 1e-6
    w[7, 5] = inf
    w[8, 5], w[8, 77] = inf, -inf
    w[9, 100] = nan
    w[10, 0] = -inf
    w[11, 127] = 60000.0
    _same(w.to(dtype), symmetric)
