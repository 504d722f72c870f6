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
    """A transposed view takes the torch statement on the same device; codes, scales and zeros must be the same bits.
    Half of the rows hold small integers, whose quotients meet the rounding boundary exactly."""
    from quantforge_b200.quantize import quantize_w4
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    w = torch.randn(N, K, device="cuda", generator=gen) * 0.05
    w[::2] = torch.randint(-15, 16, w[::2].shape, device="cuda", generator=gen).float()
    w = w.to(dtype)
    if N > 3:
        w[3, :group] = 0
    got = quantize_w4(w, group, symmetric)
    want = quantize_w4(w.t().contiguous().t(), group, symmetric)
    for a, b in zip(got, want):
        assert (a is None and b is None) or (a.dtype == b.dtype and torch.equal(a, b))


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
