"""tcgen05 kernel: the batch tile takes the width that the row count asks for (a multiple of 16, of 32 for a pair of blocks)."""
import ctypes

import pytest
import torch

import quantforge_b200 as qf
from oracle import qf_oracle as O
from quantforge_b200 import _lib
from quantforge_b200._lib import QF_PATH_GEMM

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


def _inputs(M, N, K, group, act, zeros="const"):
    d = O.make_inputs(M=1, K=K, N=N, group_size=group, act_dtype=act, seed=M + N + K)
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=gen).to(DT[act])
    z = torch.from_numpy(d["zeros"]).cuda()
    zr = {"u4": lambda: qf.pack_zeros_u4(z), "i8": lambda: z - 8, "const": lambda: None}[zeros]()
    zero_codes = {"u4": d["zeros"], "i8": d["zeros"] - 8, "const": 0 * d["zeros"] + 8}[zeros]
    w = torch.from_numpy(O.dequant(d["codes"], d["scales"], zero_codes, group, act)).cuda().double()
    return x, torch.from_numpy(d["qweight"]).cuda(), torch.from_numpy(d["scales"]).to(DT[act]).cuda(), zr, x.double() @ w.T


# fp32 sums of K exact products against 64 bits: one rounding or truncation to 2^-23 of the running sum per MMA step of 16
# products, K / 16 = 896 of them at most and each at most a few rms, mostly of both signs; one wrong weight moves an output by
# K^-1/2 rms, 8e-3 and more
TOL = 1e-4


@pytest.mark.parametrize("M,N,K,split_k", [
    (40, 256, 512, 0), (48, 256, 512, 0),                                     # single blocks of 48 rows, splits in a cluster
    (65, 384, 2304, 1), (96, 256, 2304, 3), (113, 256, 512, 0),               # up to 128 rows
    (129, 384, 2304, 1), (177, 256, 2304, 2), (256, 384, 512, 0), (513, 384, 2304, 1), (777, 128, 512, 0),
    (65, 256, 7168, 1), (97, 512, 14336, 2), (128, 256, 7168, 1),             # pairs up to 128 rows
    (129, 256, 2304, 1), (145, 512, 4608, 2), (192, 256, 2304, 1), (209, 512, 4608, 2), (270, 256, 2304, 1), (777, 768, 4096, 1),
])
@pytest.mark.parametrize("epilogue", ["none", "silu", "residual"])
def test_batch_tile_widths(M, N, K, split_k, epilogue):
    x, qw, sc, zr, lin = _inputs(M, N, K, 128, "bf16")
    res = torch.randn(M, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    epi = {"none": qf.QF_EPI_NONE, "silu": qf.QF_EPI_SILU_MUL, "residual": qf.QF_EPI_RESIDUAL_ADD}[epilogue]
    y = qf.w4a16_linear(x, qw, sc, zr, out_dtype=torch.float32, epilogue=epi, residual=res if epilogue == "residual" else None,
                        path=QF_PATH_GEMM, split_k=split_k).double()
    delta = TOL * lin.square().mean().sqrt()
    if epilogue == "silu":
        both = lin.reshape(M, N // 16, 2, 8)
        g, u = both[:, :, 0].reshape(M, N // 2), both[:, :, 1].reshape(M, N // 2)
        want = g * torch.sigmoid(g) * u
        # the slope of silu is at most 1.1, and exponential, division and product add a few roundings of the result
        bound = delta * (1.1 * u.abs() + g.abs()) + 1e-6 * want.abs()
    elif epilogue == "residual":
        want, bound = lin + res.double(), delta + 2.0 ** -23 * (lin + res.double()).abs()
    else:
        want, bound = lin, delta
    assert ((y - want).abs() <= bound).all()


@pytest.mark.parametrize("act", ["f16", "bf16"])
@pytest.mark.parametrize("layout", ["canonical", "interleaved", "tiled"])
@pytest.mark.parametrize("zeros", ["u4", "i8", "const"])
@pytest.mark.parametrize("split_k", [0, 1, 3])
def test_pairs_of_blocks_over_layouts_and_splits(act, layout, zeros, split_k):
    """K over the split decides: pairs of 160 rows with 6144 and 2048 codes, single blocks of 144 with the planner's 512."""
    M, N, K, g = 140, 512, 6144, 256
    x, qw, sc, zr, want = _inputs(M, N, K, g, act, zeros)
    lay = {"canonical": qf.QF_LAYOUT_CANONICAL, "interleaved": qf.QF_LAYOUT_INTERLEAVED, "tiled": qf.QF_LAYOUT_TILED}[layout]
    w = qw if layout == "canonical" else qf.prepack_w4(qw, layout=lay)
    d = qf.ops._make_desc(M, N, K, g, x.dtype, torch.float32, zr, 8, QF_PATH_GEMM, split_k, lay)
    split = ctypes.c_int32()
    assert _lib.load().qf_w4a16_plan(ctypes.byref(d), None, ctypes.byref(split)) == 0
    if split_k != 1:
        assert qf.ops.workspace_bytes(d) == 65536 + split.value * (160 if split_k else 144) * N * 4
    for _ in range(2):
        y = qf.w4a16_linear(x, w, sc, zr, group_size=g, out_dtype=torch.float32, weight_layout=lay, path=QF_PATH_GEMM,
                            split_k=split_k).double()
        assert (y - want).abs().max() <= TOL * want.square().mean().sqrt()
