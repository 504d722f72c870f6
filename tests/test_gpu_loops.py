"""The streaming kernels that loop (unpack of bytes at odd addresses, the interleaved prepack) at sizes around a pass of their
loops, and what keeps them and the quantise kernels at speed: loads in flight, signals to the next kernel, the right kernel."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200.quantize import quantize_w4

pytestmark = pytest.mark.gpu

PASS = 148 * 16 * 256  # elements that the largest grid takes in one step of the loop; the kernels take four steps a pass


def best_ms(fn, reps=7):
    fn()
    best = 1e9
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("n", [1, 255, 257, PASS - 1, PASS + 1, 3 * PASS + 5, 4 * PASS, 4 * PASS + 1, 9 * PASS + 77])
def test_unpack_of_bytes(n):
    packed = torch.randint(-128, 128, (n + 1,), dtype=torch.int8, device="cuda")[1:]
    want = torch.stack([packed & 15, (packed >> 4) & 15], dim=-1).flatten()
    assert torch.equal(qf.unpack_int4(packed), want)


def _in_place(words, to_canonical):
    from quantforge_b200 import _lib, ops
    assert _lib.load().qf_prepack_w4(ops._ctx(words.device), words.data_ptr(), words.data_ptr(), words.numel(), to_canonical,
                                     torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("n", [1, 255, 257, PASS - 1, PASS + 1, 3 * PASS + 5, 4 * PASS, 4 * PASS + 1, 9 * PASS + 77])
def test_interleaved_prepack(n):
    """The even nibbles of a word in its low half, the odd ones in its high half; and back, also in place."""
    words = torch.randint(-2 ** 31, 2 ** 31 - 1, (1, n), dtype=torch.int32, device="cuda")
    want = torch.zeros(1, n, dtype=torch.int64, device="cuda")
    for j in range(8):
        want |= ((words.long() >> 4 * j) & 15) << (4 * (j // 2) + 16 * (j % 2))
    out = qf.prepack_w4(words)
    assert torch.equal(out.long() & 0xffffffff, want)
    assert torch.equal(qf.prepack_w4(out, to_canonical=True), words)
    _in_place(words, 0)
    assert torch.equal(words, out)
    _in_place(words, 1)
    assert torch.equal(qf.prepack_w4(words), out)


def test_loops_keep_several_loads_in_flight():
    """A byte at a time takes 1.6 times the time of whole vectors and the interleaved prepack 1.2 times that of the tiled one;
    with one load in flight per thread it is 3.6 and 1.8 times."""
    n = 64 << 20
    flat = torch.randint(-128, 128, (n + 16,), dtype=torch.int8, device="cuda")
    odd, even = best_ms(lambda: qf.unpack_int4(flat[1:n + 1])), best_ms(lambda: qf.unpack_int4(flat[:n]))
    assert odd < 2.1 * even
    w = torch.randint(-128, 128, (28672, 4096), dtype=torch.int8, device="cuda")
    inter, tiled = best_ms(lambda: qf.prepack_w4(w)), best_ms(lambda: qf.prepack_w4(w, layout=qf.QF_LAYOUT_TILED))
    assert inter < 1.45 * tiled


@pytest.mark.parametrize("symmetric", [False, True])
def test_small_groups_are_not_bound_by_their_blocks_signals(symmetric):
    """Groups of 256, a block of 64 threads each, take about the time of groups of 1024 in blocks of 256; 1.8 times that when
    every block signals the next kernel."""
    w = (torch.randn(4096, 14336, device="cuda") * 0.02).to(torch.bfloat16)
    small, large = (best_ms(lambda: quantize_w4(w, g, symmetric)) for g in (256, 1024))
    assert small < 1.35 * large


@pytest.mark.parametrize("N", [65535 * 16 - 1, 65535 * 16 + 1, 2 * 65535 * 16 + 33])
@pytest.mark.parametrize("symmetric", [False, True])
def test_quantise_more_than_65535_blocks_of_rows(N, symmetric):
    """The rows of a tall matrix, in groups of 128, are the rows of its parts."""
    w = torch.randn(N, 128, device="cuda").mul_(0.02).to(torch.bfloat16)
    codes, scales, zeros = quantize_w4(w, 128, symmetric)
    for a, b in ((0, 500000), (500000, 65535 * 16 - 40), (65535 * 16 - 40, N)):
        for c0 in range(a, b, 1000000):
            c1 = min(b, c0 + 1000000)
            c, s, z = quantize_w4(w[c0:c1], 128, symmetric)
            assert torch.equal(codes[c0:c1], c) and torch.equal(scales[:, c0:c1], s)
            assert symmetric or torch.equal(zeros[:, c0:c1], z)


def test_tall_matrices_take_the_same_kernel():
    """1.1 million rows take about as long a row as 1.0 million; a block per group took three times that."""
    w = torch.randn(1100000, 128, device="cuda").mul_(0.02).to(torch.bfloat16)
    tall, lower = best_ms(lambda: quantize_w4(w, 128)), best_ms(lambda: quantize_w4(w[:1000000], 128))
    assert tall < 1.3 * lower
