"""Quantise in groups that are a thread block each: both ends of what each size of block takes, in one tile and in several."""
import pytest
import torch

from test_gpu_quantize_quotients import _same

pytestmark = pytest.mark.gpu


# 64, 128, 192, 256, 320, 384, 448 and 512 threads of 16 values; two tiles of 320 to 512, three of 384 and 512, four of 512
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("group", [528, 1024, 1040, 2048, 2064, 3072, 3088, 4096, 4112, 5120, 5136, 6144, 6160, 7168, 7184, 8192, 8208, 10240, 10256, 12288,
                                   12304, 14336, 14352, 16384, 16400, 18432, 18448, 24576, 28672, 32768])
def test_blocks(group, dtype):
    gen = torch.Generator(device="cuda").manual_seed(group)
    w = (torch.randn(3, 2 * group, device="cuda", generator=gen) * 0.05).to(dtype)
    for at, value in ((0, 0.5), (group - 1, -0.5), (group, 1.0), (2 * group - 1, float("nan"))):
        w[1, at] = value
    w[2, :group] = 0.0
    for symmetric in (False, True):
        _same(w, group, symmetric)
