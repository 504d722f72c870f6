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


@pytest.mark.parametrize("M,K,N", [(4, 14336, 1040), (16, 4096, 4112), (64, 28672, 4112), (200, 14336, 1040), (777, 4096, 4176)])
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
