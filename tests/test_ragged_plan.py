"""Which kernel AUTO picks for canonical weights whose rows are no multiple of 128 (host logic of qf_w4a16_plan). No GPU needed."""
import ctypes

import pytest

from quantforge_b200 import _lib
from quantforge_b200._lib import QF_PATH_AUTO, QF_PATH_GEMM, QF_PATH_GEMV


def _desc(M, K, N, path=QF_PATH_AUTO, split_k=0, zero_mode=_lib.QF_ZERO_I8, out_dtype=_lib.QF_BF16):
    return _lib.LinearDesc(M=M, N=N, K=K, group_size=128, act_dtype=_lib.QF_BF16, out_dtype=out_dtype, zero_mode=zero_mode, zero_const=8,
                           path=path, split_k=split_k)


def _plan(*args, **kw):
    """(path, split), or the status of a refused descriptor."""
    d, path, split = _desc(*args, **kw), ctypes.c_int32(), ctypes.c_int32()
    st = _lib.load().qf_w4a16_plan(ctypes.byref(d), ctypes.byref(path), ctypes.byref(split))
    return st if st != 0 else (path.value, split.value)


@pytest.mark.parametrize("M,K,N", [(4, 8192, 4112), (16, 4096, 4112), (64, 28672, 4112), (200, 14336, 1040), (777, 4096, 4176)])
def test_named_splits_are_those_of_the_gemv_kernel(M, K, N):
    assert _plan(M, K, N)[0] == QF_PATH_GEMM
    for split in (1, 2, 3, 8, 16, 100):
        assert _plan(M, K, N, split_k=split) == _plan(M, K, N, path=QF_PATH_GEMV, split_k=split)


# the GEMV kernel's tiles of 64 columns x 8 rows: 449 x 37 and 38, 16385 x 1 (16384 have a counter)
@pytest.mark.parametrize("M,K,N,refused", [(296, 8192, 28688, True), (288, 8192, 28688, False), (300, 4096, 28688, False), (8, 4224, 1048640 - 48, True),
                                           (8, 4096, 1048640 - 48, False), (8, 4224, 1048640 - 64, False)])
def test_what_the_gemv_kernel_refuses_stays_refused(M, K, N, refused):
    for out_dtype in (_lib.QF_BF16, _lib.QF_F32):
        for path in (QF_PATH_AUTO, QF_PATH_GEMV):
            assert (_plan(M, K, N, path=path, out_dtype=out_dtype) == -2) == refused  # QF_ERR_UNSUPPORTED


def _gemm(M, K, N, **kw):
    return _plan(M, K, N, **kw)[0] == QF_PATH_GEMM


# on either side of each line, by rows of activations: (rows, K, largest N of the GEMV kernel, smallest of the tcgen05 kernel)
@pytest.mark.parametrize("rows,K,gemv,gemm", [
    ((3, 4), 896, 40976, None), ((3, 4), 1024, 12272, 12304), ((3, 4), 1408, 12272, 12304), ((3, 4), 1536, 7792, 7824), ((3, 4), 2432, 4912, 4944),
    ((3, 4), 2560, 3888, 3920), ((3, 4), 4096, 2416, 2448), ((3, 4), 4480, 2224, 2256), ((3, 4), 4608, 1296, 1328), ((3, 4), 5120, 1936, 1968),
    ((3, 4), 5248, 1136, 1168), ((3, 4), 12288, 464, 496), ((3, 4), 14208, 400, 432), ((3, 4), 14336, 2672, 2704), ((3, 4), 28672, 2672, 2704),
    ((5, 6, 7, 8), 896, 40976, None), ((5, 6, 7, 8), 1024, 12176, 12208), ((5, 6, 7, 8), 1536, 5200, 5232), ((5, 6, 7, 8), 2560, 2320, 2352),
    ((5, 6, 7, 8), 14336, 400, 432), ((5, 6), 20480, 272, 304), ((5, 6), 20608, 1520, 1552), ((7, 8), 24576, 240, 272),
    ((9, 12, 16), 512, 7792, 7824), ((9, 16), 640, 19504, 19536), ((9, 16), 896, 10032, 10064), ((9, 16), 1024, 3888, 3920), ((9, 12, 16), 4096, 976, 992), ((9, 16), 28672, 112, 144),
    ((17, 24), 512, 3888, 3920), ((17, 24), 128, 19504, 19536), ((25, 40), 128, 15600, 15632), ((17, 40), 256, 9744, 9776), ((41, 64), 256, 7792, 7824), ((17, 24), 640, 14048, 14096), ((17, 24), 1024, 3888, 3920), ((17, 24), 1408, 3184, 3216), ((17, 24), 896, 7792, 7824), ((17, 24, 32, 40, 64), 1536, 1296, 1328),
    ((25, 32), 896, 4432, 4496), ((25, 32), 640, 9360, 9392), ((33, 40), 640, 7792, 7824), ((41, 64), 640, 6224, 6256), ((25, 32), 1024, 1936, 1968), ((25, 32), 1280, 2288, 2320), ((33, 40), 1024, 2320, 2352), ((41, 64), 1024, 1936, 1968),
    ((17, 32), 28672, 48, 80), ((33, 40), 28672, 240, 272), ((33, 40), 20480, 144, 176), ((41, 56), 28672, 144, 176), ((57, 64), 28672, 112, 144),
    ((65, 79), 1024, 5072, 5104), ((80, 128), 1024, 3888, 3920), ((65, 79), 2048, 1936, 1968), ((81, 104), 2048, 2192, 2224), ((105, 256), 2048, 1936, 1968),
    ((96, 128), 14336, 496, 528), ((160,), 14336, 400, 432), ((65, 256), 28672, 144, None), ((112,), 28672, 272, 304), ((140,), 28672, 208, 240),
    ((257, 777), 28672, 112, 144), ((257, 777), 4096, 976, 992), ((64,), 8192, 240, 272), ((65,), 8192, 480, 496),
])
def test_lines(rows, K, gemv, gemm):
    for M in rows:
        assert not _gemm(M, K, gemv)
        for N in (gemm, gemm + 16, gemm + 4096 + 16) if gemm else ():
            assert N % 128 == 0 or _gemm(M, K, N), (M, N)
        # one or two rows, and results whose sums are not rounded: the other kernel
        for N in (gemv, gemm or gemv):
            assert not _gemm(1, K, N) and not _gemm(2, K, N) and not _gemm(M, K, N, out_dtype=_lib.QF_F32)


@pytest.mark.parametrize("M", [3, 8, 16, 64, 200])
def test_packed_zeros_come_in_multiples_of_sixteen_bytes(M):
    # four bits a zero: 16 bytes are 32 columns, so what is left for the last tile is a multiple of that (or there are no zeros in memory)
    for N in range(5136, 5136 + 128, 16):
        if N % 128:
            assert _gemm(M, 4096, N, zero_mode=_lib.QF_ZERO_U4) == (N % 32 == 0)
            assert _gemm(M, 4096, N) and _gemm(M, 4096, N, zero_mode=_lib.QF_ZERO_CONST)
