"""Launch planning (host logic of qf_w4a16_plan): which kernel AUTO picks and how K is split. No GPU needed."""
import ctypes

import pytest

from quantforge_b200 import _lib


def _plan(M, K, N, layout=0, path=0, split_k=0):
    lib = _lib.load()
    d = _lib.LinearDesc(M=M, N=N, K=K, group_size=128, act_dtype=_lib.QF_BF16, out_dtype=_lib.QF_BF16,
                        zero_mode=_lib.QF_ZERO_U4, zero_const=8, path=path, split_k=split_k, weight_layout=layout)
    pa, sk = ctypes.c_int32(), ctypes.c_int32()
    st = lib.qf_w4a16_plan(ctypes.byref(d), ctypes.byref(pa), ctypes.byref(sk))
    assert st == 0
    return pa.value, sk.value


@pytest.mark.parametrize("M,K,N,layout,want", [
    (1, 4096, 4096, 0, _lib.QF_PATH_GEMV),        # small matrix, decode batch 1
    (2, 4096, 14336, 0, _lib.QF_PATH_GEMV),       # 29 MB: still the GEMV kernel
    (3, 4096, 4096, 0, _lib.QF_PATH_GEMM),        # M >= 3: tcgen05
    (1, 4096, 4096, 1, _lib.QF_PATH_GEMM),        # prepacked weights are read by the tcgen05 kernel only
    (1, 8192, 8192, 1, _lib.QF_PATH_GEMM),        # 32 MB prepacked: tcgen05
    (1, 8192, 8192, 0, _lib.QF_PATH_GEMV),        # 32 MB canonical: below the 40 MB crossover
    (1, 4096, 28672, 0, _lib.QF_PATH_GEMM),       # 56 MB canonical: tcgen05
    (1, 28672, 8192, 1, _lib.QF_PATH_GEMM),
    (16, 4096, 144, 0, _lib.QF_PATH_GEMV),        # N not a multiple of 128: only the GEMV kernel can
    (1, 16384, 4112, 0, _lib.QF_PATH_GEMV),       # large but N % 128 != 0
])
def test_auto_path(M, K, N, layout, want):
    assert _plan(M, K, N, layout)[0] == want


def test_forced_paths_are_respected():
    assert _plan(1, 8192, 57344, 0, path=_lib.QF_PATH_GEMV)[0] == _lib.QF_PATH_GEMV
    assert _plan(1, 4096, 4096, 0, path=_lib.QF_PATH_GEMM)[0] == _lib.QF_PATH_GEMM
    assert _plan(16, 4096, 4096, 1, split_k=3) == (_lib.QF_PATH_GEMM, 3)


def test_even_k_splits_are_preferred():
    # K = 14336 = 112 k-blocks of 128, 32 tiles: 296 block slots / 32 = 9 splits would leave a short last split
    assert _plan(16, 14336, 4096, 1) == (_lib.QF_PATH_GEMM, 8)
    assert _plan(64, 14336, 4096, 1) == (_lib.QF_PATH_GEMM, 8)
    # GEMV kernel: 112 chunks, 64 column blocks -> 9 splits by block count, 8 divides K evenly and fits a cluster
    assert _plan(1, 14336, 4096, 0) == (_lib.QF_PATH_GEMV, 8)
    # 4096 x 14336: 112 tiles, two splits fill the device
    assert _plan(16, 4096, 14336, 1) == (_lib.QF_PATH_GEMM, 2)


def test_no_split_when_tiles_fill_the_device():
    assert _plan(2048, 8192, 28672, 1) == (_lib.QF_PATH_GEMM, 1)
    assert _plan(64, 8192, 28672, 1) == (_lib.QF_PATH_GEMM, 1)


def test_splits_stay_within_one_wave_of_clusters():
    # tcgen05 kernel, narrow tiles: at most 8 splits and at most 256 blocks, so that the split-K sum stays on chip
    assert _plan(16, 4096, 6144, 1) == (_lib.QF_PATH_GEMM, 5)     # 48 tiles: 6 splits would be 288 blocks
    assert _plan(64, 4096, 5120, 1) == (_lib.QF_PATH_GEMM, 6)     # 40 tiles
    assert _plan(16, 8192, 1024, 1) == (_lib.QF_PATH_GEMM, 8)     # 8 tiles: not 16 splits through global memory
    assert _plan(16, 8192, 10240, 1) == (_lib.QF_PATH_GEMM, 3)    # 80 tiles
    assert _plan(16, 4096, 18944, 1) == (_lib.QF_PATH_GEMM, 2)    # 148 tiles: two splits fill every slot


def _tile_rows(M, K, N, split_k=0):
    """Batch tile width of a split tcgen05 launch, from its scratch: counters, then split x tiles x width x N floats."""
    d = _lib.LinearDesc(M=M, N=N, K=K, group_size=128, act_dtype=_lib.QF_BF16, out_dtype=_lib.QF_BF16,
                        zero_mode=_lib.QF_ZERO_U4, zero_const=8, path=_lib.QF_PATH_GEMM, split_k=split_k, weight_layout=2)
    split = _plan(M, K, N, 2, _lib.QF_PATH_GEMM, split_k)[1]
    assert split > 1
    floats = (_lib.load().qf_w4a16_workspace_bytes(ctypes.byref(d)) - 16384 * 4) // 4
    tiles = (M + 255) // 256
    assert floats % (split * tiles * N) == 0
    return floats // (split * tiles * N)


@pytest.mark.parametrize("M,K,N,split_k,want", [
    # a multiple of 32: a pair of blocks; of 16 only: single blocks
    (72, 4096, 1024, 0, 80),       # 512 codes a block
    (72, 14336, 4096, 0, 80),      # 3584
    (72, 28672, 4096, 0, 96),      # 7168
    (72, 14336, 4096, 2, 96),
    (140, 4096, 4096, 0, 144),     # 1024
    (140, 8192, 4096, 0, 160),     # 2048
    (140, 6144, 4096, 0, 160),     # 1536
    (140, 8192, 4096, 8, 144),
    (200, 8192, 1024, 0, 208),     # 512
    (200, 8192, 4096, 0, 208),     # 2048
    (200, 14336, 4096, 0, 224),    # 3584
    (1030, 6144, 1024, 0, 208),    # five tiles of 206 rows, 2048 codes
    (200, 14336, 4224, 0, 208),    # N no multiple of 256
])
def test_pairs_where_a_block_runs_through_enough_codes(M, K, N, split_k, want):
    assert _tile_rows(M, K, N, split_k) == want


@pytest.mark.parametrize("M", [16, 72, 140, 256])
def test_blocks_take_512_codes_at_least(M):
    for K in (512, 1024, 2048, 4096):
        assert K // _plan(M, K, 1024, 2, _lib.QF_PATH_GEMM)[1] >= 512


@pytest.mark.parametrize("K,N", [(128, 64), (4096, 4096), (8192, 28672), (5760, 57344), (8192, 57344), (28672, 11520), (28672, 28672)])
def test_up_to_8_rows_one_kernel_reads_slab_weights(K, N):
    # AUTO is the streaming GEMV kernel, which QF_PATH_GEMV names, at any size: one order of sums for all of them
    for M in range(1, 9):
        assert _plan(M, K, N, _lib.QF_LAYOUT_GEMV_SLAB) == _plan(M, K, N, _lib.QF_LAYOUT_GEMV_SLAB, _lib.QF_PATH_GEMV)


def _slab_desc(M, K, N):
    return _lib.LinearDesc(M=M, N=N, K=K, group_size=128, act_dtype=_lib.QF_BF16, out_dtype=_lib.QF_BF16, zero_mode=_lib.QF_ZERO_U4,
                           zero_const=8, weight_layout=_lib.QF_LAYOUT_GEMV_SLAB)


def _row_tiles(M):
    return 1 if M <= 8 else 2 if M <= 16 else 4


@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16, 17, 32])
def test_scratch_of_a_slab_linear_is_that_of_its_own_kernels(M):
    """What one call on a descriptor can reach: the kernel of the plan and an exchange's launch. Chains are asked for by the batch."""
    lib = _lib.load()
    for K, N in ((128, 64), (512, 512), (2048, 1024), (2560, 1024), (4096, 4096), (4096, 14336), (8192, 57344)):
        blob = N // 64 * (K // 128) * 4352
        units = blob // 4352
        blocks = min(units, 148 * (2 if blob <= 16 << 20 else 3 if M > 16 else 4))
        words = blocks * 4 * _row_tiles(M) * 128  # a tile of partial sums per warp
        tcgen05 = M > 8 and _plan(M, K, N, _lib.QF_LAYOUT_GEMV_SLAB) != _plan(M, K, N, _lib.QF_LAYOUT_GEMV_SLAB, _lib.QF_PATH_GEMV)
        if tcgen05:  # its counters and slots, four a block
            words = max(words, 8192 + 4 * 148 * ((M + 1) // 2 * 2) * 128)
        d = _slab_desc(M, K, N)
        assert lib.qf_w4a16_workspace_bytes(ctypes.byref(d)) == 8 * words
    if M <= 8:  # fits what the package makes for a stream at first
        assert lib.qf_w4a16_workspace_bytes(ctypes.byref(_slab_desc(M, 28672, 57344))) <= 4 << 20


def test_scratch_of_a_batch():
    lib = _lib.load()

    def need(*descs):
        return lib.qf_w4a16_batched_workspace_bytes(len(descs), (_lib.LinearDesc * len(descs))(*descs))

    alone = lambda d: lib.qf_w4a16_workspace_bytes(ctypes.byref(d))  # noqa: E731
    small, large = _slab_desc(1, 1024, 1024), _slab_desc(1, 4096, 14336)
    assert need(small) == alone(small) and need() == 0
    assert need(small, large) == 65536 + 2 * 4 * 148 * 4096
    many = _slab_desc(32, 128, 128)
    assert need(many) == alone(many) == 4 * 4096 * 2 and need(many, many) == 65536 + 4 * 148 * 32 * 128 * 8
    # what does not chain: other rows, half row blocks above 8 rows
    assert need(small, _slab_desc(2, 1024, 1024)) == alone(small)
    half = _slab_desc(9, 1024, 64)
    assert need(half, half) == alone(half)


@pytest.mark.parametrize("M,K,mib,tcgen05", [
    # up to 16 rows; the GEMV kernel's time is up to 1.3 times the other's where this says False, and the other way round
    (9, 14336, 25, True), (16, 8192, 25, True), (9, 8192, 22, False), (16, 6144, 35, True), (9, 6144, 30, False), (12, 5120, 44, True),
    (16, 5120, 34, False), (16, 4096, 48, False), (9, 4096, 34, False), (16, 1024, 34, False), (9, 2048, 64, False), (16, 4096, 74, True),
    (9, 512, 74, True), (9, 256, 120, False),
    (17, 3072, 25, True), (32, 14336, 25, True), (32, 4096, 22, False), (17, 2048, 25, False), (24, 1024, 36, True), (32, 1024, 36, False),
    (32, 512, 44, True),
])
def test_which_kernel_reads_large_slab_weights(M, K, mib, tcgen05):
    N = round(mib * 2 ** 20 / 4352 / (K // 128)) * 64
    auto, gemv = (_plan(M, K, N, _lib.QF_LAYOUT_GEMV_SLAB, path) for path in (_lib.QF_PATH_AUTO, _lib.QF_PATH_GEMV))
    # the tcgen05 kernel divides the weights among two streams of each SM whatever the size is
    assert gemv[1] != 296 and (auto == (_lib.QF_PATH_GEMV, 296) if tcgen05 else auto == gemv)
