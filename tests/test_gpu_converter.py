"""The register converters of the linear kernels (packed codes to 16-bit weights), weight by weight.

With the rows of an identity matrix as activations and fp32 results, a linear returns its weights: one product by 1 and zeros
otherwise. They must be the bits `dequant_w4` writes, whose kernel does not use the converter of the tcgen05 kernel."""
import pytest
import torch

import quantforge_b200 as qf
from quantforge_b200._lib import QF_PATH_GEMM, QF_PATH_GEMV

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


def _weights(act, zeros, N=512, K=128):
    """All codes, all zero points, scales over the exponents of the type (products that are finite, normal fp32 numbers)."""
    gen = torch.Generator().manual_seed(0)
    qw = torch.randint(-128, 128, (N, K // 2), dtype=torch.int8, generator=gen)
    lo, hi = (-24, 8) if act == "f16" else (-120, 119)
    e = torch.randint(lo, hi, (1, N), generator=gen).double()
    sc = ((1 + torch.rand(1, N, generator=gen, dtype=torch.float64)) * 2.0 ** e).to(DT[act])
    n = torch.arange(N)
    if zeros == "u4":
        zr = qf.pack_zeros_u4((n % 16).to(torch.int8).reshape(1, N).cuda())
    else:
        zr = (n % 256 - 128).to(torch.int8).reshape(1, N).cuda()
    return qw.cuda(), sc.cuda(), zr


def _through_linear(act, layout, M, qw, sc, zr):
    K = qw.shape[1] * 2
    kw = {}
    if layout == "slab":
        w = (qf.prepack_gemv_slab(qw, sc, zr, group_size=K),)
    elif layout in ("gemv", "canonical"):
        w, kw = (qw, sc, zr), {"group_size": K, "path": QF_PATH_GEMV if layout == "gemv" else QF_PATH_GEMM}
    else:
        lay = qf.QF_LAYOUT_INTERLEAVED if layout == "interleaved" else qf.QF_LAYOUT_TILED
        w, kw = (qf.prepack_w4(qw, layout=lay), sc, zr), {"group_size": K, "weight_layout": lay}
    eye = torch.eye(K, dtype=DT[act], device="cuda")
    return torch.cat([qf.w4a16_linear(eye[k:k + M].contiguous(), *w, out_dtype=torch.float32, **kw) for k in range(0, K, M)]).T


@pytest.mark.parametrize("act", ["f16", "bf16"])
@pytest.mark.parametrize("zeros", ["u4", "i8"])
@pytest.mark.parametrize("layout,M", [("slab", 1), ("slab", 8), ("slab", 32), ("gemv", 1), ("gemv", 8), ("canonical", 16),
                                      ("interleaved", 128), ("tiled", 64)])
def test_linear_of_identity_returns_the_weights(act, zeros, layout, M):
    qw, sc, zr = _weights(act, zeros)
    want = qf.dequant_w4(qw, sc, zr, group_size=128).float()
    assert torch.isfinite(want).all()
    assert torch.equal(_through_linear(act, layout, M, qw, sc, zr), want)


@pytest.mark.parametrize("layout,M", [("slab", 1), ("canonical", 16), ("tiled", 128)])
def test_scales_at_the_end_of_the_bf16_range(layout, M):
    """Scales of 2^126 and more, whose fourfold is infinite, beside small ones; codes at and next to the zero point."""
    gen = torch.Generator().manual_seed(1)
    N, K = 256, 128
    codes = torch.randint(7, 10, (N, K), dtype=torch.uint8, generator=gen)
    qw = qf.pack_int4(codes.to(torch.int8).cuda())
    sc = torch.where(torch.arange(N) % 3 == 0, 1.5 * 2.0 ** 126, 2.0 ** -100).to(torch.bfloat16).reshape(1, N).cuda()
    want = qf.dequant_w4(qw, sc, None, group_size=K).float()
    assert torch.isfinite(want).all()
    assert torch.equal(_through_linear("bf16", layout, M, qw, sc, None), want)
