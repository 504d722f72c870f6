"""tcgen05 kernel: the batch tile takes the width that the row count asks for (a multiple of 16, of 32 for a pair of blocks)."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200._lib import QF_PATH_GEMM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [48, 49, 65, 80, 81, 113, 129, 144, 145, 177, 209, 257, 270, 289, 513, 777])
# K above 2048 with N a multiple of 256: pairs of blocks
@pytest.mark.parametrize("N,K", [(256, 512), (256, 2304), (384, 2304), (768, 4096)])
@pytest.mark.parametrize("epilogue", ["none", "silu", "residual"])
def test_batch_tile_widths(M, N, K, epilogue):
    """Results as those of 64 rows at a time."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.rand(K // 128, N, device="cuda", generator=gen) * 0.01 + 0.001).bfloat16()
    x = torch.randn(M, K, device="cuda", generator=gen).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=gen)
    epi = {"none": qf.QF_EPI_NONE, "silu": qf.QF_EPI_SILU_MUL, "residual": qf.QF_EPI_RESIDUAL_ADD}[epilogue]

    def call(a, r):
        return qf.w4a16_linear(a, qw, sc, None, out_dtype=torch.float32, epilogue=epi,
                               residual=r if epilogue == "residual" else None, path=QF_PATH_GEMM)

    y = call(x, res)
    want = torch.cat([call(x[i:i + 64].contiguous(), res[i:i + 64].contiguous()) for i in range(0, M, 64)])
    # fp32 sums of K products in another order: K * 2^-24 of the sum of magnitudes, which is below sqrt(K) rms of a sum; a
    # SiLU * mul output adds the errors of two of them, each times the other's value of at most 5 rms
    tol = K * 2.0 ** -24 * K ** 0.5 * 10 * want.square().mean().sqrt()
    assert (y - want).abs().max() <= tol


@pytest.mark.parametrize("act", ["f16", "bf16"])
@pytest.mark.parametrize("layout", ["canonical", "interleaved", "tiled"])
@pytest.mark.parametrize("zeros", ["u4", "i8", "const"])
@pytest.mark.parametrize("split_k", [0, 1, 3])
def test_pairs_of_blocks_over_layouts_and_splits(act, layout, zeros, split_k):
    """The paired kernel against the unpaired one (64 rows at a time): the same sums of exactly rounded weights."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    dt = {"f16": torch.float16, "bf16": torch.bfloat16}[act]
    M, N, K, g = 150, 512, 3072, 256
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, device="cuda", generator=gen)
    sc = (torch.rand(K // g, N, device="cuda", generator=gen) * 0.01 + 0.001).to(dt)
    z = torch.randint(0, 16, (K // g, N), dtype=torch.int8, device="cuda", generator=gen)
    zr = {"u4": lambda: qf.pack_zeros_u4(z), "i8": lambda: z - 8, "const": lambda: None}[zeros]()
    lay = {"canonical": qf.QF_LAYOUT_CANONICAL, "interleaved": qf.QF_LAYOUT_INTERLEAVED, "tiled": qf.QF_LAYOUT_TILED}[layout]
    w = qw if layout == "canonical" else qf.prepack_w4(qw, layout=lay)
    x = torch.randn(M, K, device="cuda", generator=gen).to(dt)

    def call(a, split):
        return qf.w4a16_linear(a, w, sc, zr, group_size=g, out_dtype=torch.float32, weight_layout=lay, path=QF_PATH_GEMM,
                               split_k=split)

    want = torch.cat([call(x[i:i + 50].contiguous(), 1) for i in range(0, M, 50)])
    tol = K * 2.0 ** -24 * K ** 0.5 * want.square().mean().sqrt()  # another order of the same fp32 sums, as above
    for _ in range(2):
        assert (call(x, split_k) - want).abs().max() <= tol
