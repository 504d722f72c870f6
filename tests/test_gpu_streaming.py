"""The streaming kernels around the linears at the sizes where they can go wrong: quantise, pack, unpack and dequant,
bit for bit against the plain torch statement or the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import qf_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,group", [(1, 128, 128), (33, 384, 128), (64, 1024, 256), (7, 1152, 1152), (40, 96, 12), (5, 2048, 2048)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("symmetric", [False, True])
def test_quantise_kernel_is_the_torch_statement(N, K, group, dtype, symmetric):
    """A weight that requires grad takes the torch statement on the same device; codes, scales and zeros must be the same bits.
    Half of the rows hold small integers, whose quotients meet the rounding boundary exactly."""
    import quantforge_b200 as qf
    from quantforge_b200.quantize import quantize_w4
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    w = torch.randn(N, K, device="cuda", generator=gen) * 0.05
    w[::2] = torch.randint(-15, 16, w[::2].shape, device="cuda", generator=gen).float()
    w = w.to(dtype)
    if N > 3:
        w[3, :group] = 0
    got = quantize_w4(w, group, symmetric)
    before = qf.launch_count()
    want = quantize_w4(w.clone().requires_grad_(), group, symmetric)
    assert qf.launch_count() == before
    for a, b in zip(got, want):
        assert (a is None and b is None) or (a.dtype == b.dtype and torch.equal(a, b))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("symmetric", [False, True])
def test_quantise_kernel_and_cpu(dtype, symmetric):
    """The CPU divides where CUDA multiplies with the reciprocal: scales are the same 16-bit number or its neighbour, and
    under the same scale codes and zeros are the same."""
    from quantforge_b200.quantize import quantize_w4
    w = (torch.randn(512, 4096, generator=torch.Generator().manual_seed(5)) * 0.05).to(dtype)
    codes, scales, zeros = quantize_w4(w.cuda(), 128, symmetric)
    c, s, z = quantize_w4(w, 128, symmetric)
    ulps = (scales.cpu().view(torch.int16).int() - s.view(torch.int16).int()).abs()
    assert ulps.max() <= 1 and (ulps > 0).float().mean() < 2e-3
    same = ulps == 0
    assert zeros is None or torch.equal(zeros.cpu()[same], z[same])
    rows = same.t().repeat_interleave(128, dim=1)
    assert torch.equal(codes.cpu()[rows], c[rows])


@pytest.mark.parametrize("shape", [(1, 2), (3, 10), (5, 48), (33, 998), (4096, 2048), (2, 3, 64)])
def test_pack_kernel(shape):
    import quantforge_b200 as qf
    codes = np.random.default_rng(sum(shape)).integers(-128, 128, size=shape, dtype=np.int8)  # upper bits are ignored
    got = qf.pack_int4(torch.from_numpy(codes).cuda())
    assert np.array_equal(got.cpu().numpy(), O.pack_int4(codes & 0xF))
    assert np.array_equal(qf.unpack_int4(got).cpu().numpy(), codes & 0xF)


@pytest.mark.parametrize("G,N", [(1, 8), (3, 40), (32, 4096)])
def test_pack_zeros_kernel(G, N):
    import quantforge_b200 as qf
    z = np.random.default_rng(G).integers(0, 16, size=(G, N), dtype=np.int8)
    got = qf.pack_zeros_u4(torch.from_numpy(z).cuda())
    assert np.array_equal(got.cpu().numpy().view(np.uint32), O.pack_zeros_u4(z))


@pytest.mark.parametrize("N,K,group", [(16, 128, 128), (48, 640, 128), (80, 1024, 512), (16, 4224, 4224)])
@pytest.mark.parametrize("act", ["f16", "bf16"])
def test_dequant_ragged(N, K, group, act):
    import quantforge_b200 as qf
    d = O.make_inputs(M=1, K=K, N=N, group_size=group, act_dtype=act, seed=N + K)
    want = O.dequant(d["codes"], d["scales"], d["zeros"], group, act)
    dt = torch.float16 if act == "f16" else torch.bfloat16
    got = qf.dequant_w4(torch.from_numpy(d["qweight"]).cuda(), torch.from_numpy(d["scales"]).to(dt).cuda(),
                        qf.pack_zeros_u4(torch.from_numpy(d["zeros"]).cuda()), group)
    assert np.array_equal(got.float().cpu().numpy(), want)


def _unpack_into(packed, out):
    from quantforge_b200 import _lib, ops
    ctx = ops._ctx(packed.device)
    st = _lib.load().qf_unpack_int4(ctx, packed.data_ptr(), out.data_ptr(), 1, packed.numel(),
                                    torch.cuda.current_stream().cuda_stream)
    assert st == 0


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4096, 70001])
@pytest.mark.parametrize("offset", [0, 2, 16, 32, 48])
@pytest.mark.parametrize("shift", [0, 1])
def test_unpack_at_any_alignment(n, offset, shift):
    """Through the C entry: outputs aligned to 32, 16 and 2 bytes, inputs to 16 and 1; nothing written beside them."""
    packed = torch.from_numpy(np.random.default_rng(n).integers(-128, 128, size=n + shift, dtype=np.int8)).cuda()[shift:]
    buf = torch.full((2 * n + 128,), 77, dtype=torch.int8, device="cuda")
    _unpack_into(packed, buf[offset:offset + 2 * n])
    got = buf.cpu().numpy()
    assert np.array_equal(got[offset:offset + 2 * n], O.unpack_int4(packed.cpu().numpy().reshape(1, -1))[0])
    assert (got[:offset] == 77).all() and (got[offset + 2 * n:] == 77).all()


def test_unpack_of_sixteen_byte_aligned_outputs_is_no_byte_loop():
    """An output that starts in the middle of a 32-byte sector takes the vector kernel too, and stores whole sectors: 0.98 times the time of
    an aligned one (31.9 against 32.4 us in calls behind one another), where half sectors take 1.24 times (40.3 us) and a byte per
    thread 1.75 times."""
    n = 64 << 20
    packed = torch.randint(-128, 128, (n,), dtype=torch.int8, device="cuda")
    buf = torch.empty(2 * n + 16, dtype=torch.int8, device="cuda")

    def ms(out):
        # (twenty behind one another: the first call finds some of its input in L2)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(20):
            _unpack_into(packed, out)
        b.record()
        b.synchronize()
        return a.elapsed_time(b)

    times = [(ms(buf[:2 * n]), ms(buf[16:])) for _ in range(12)]
    aligned, half = (min(t) for t in zip(*times))
    assert half < 1.12 * aligned


def test_dequant_of_very_long_rows():
    """More than 65535 blocks of columns (33.5 million codes a row)."""
    import quantforge_b200 as qf
    N, K, group = 16, 512 * 65537, 512 * 65537
    g = torch.Generator(device="cuda").manual_seed(0)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=g)
    sc = (torch.rand(1, N, device="cuda", generator=g) * 0.01 + 0.001).half()
    got = qf.dequant_w4(qw, sc, None, group)
    for n in range(N):
        codes = torch.stack([qw[n] & 15, (qw[n] >> 4) & 15], dim=-1).flatten()
        assert torch.equal(got[n], (codes - 8).half() * sc[0, n])  # a difference that is exact and one rounding
