// C ABI of the runtime (include/quantforge_rt.h): argument checks, planning, dispatch.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <new>

#include <cuda.h>

#include "qf_common.cuh"
#include "qf_stream.cuh"

namespace qf {

std::atomic<long long> g_launch_count{0};

bool pdl_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("QF_PDL");
        return !(e && e[0] == '0');
    }();
    return on;
}

// The node that a stream in capture depends on, where it is a single one.
static bool capture_tail(cudaStream_t s, unsigned long long *id, cudaGraphNode_t *node) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    const cudaGraphNode_t *deps = nullptr;
    const cudaGraphEdgeData *edges = nullptr;
    size_t n = 0;
    if (cudaStreamGetCaptureInfo_v3(s, &status, id, nullptr, &deps, &edges, &n) != cudaSuccess) {
        cudaGetLastError();  // the launch says what is wrong with the stream
        return false;
    }
    if (status != cudaStreamCaptureStatusActive || n != 1) return false;
    *node = deps[0];
    return true;
}

// The linear that this thread captured last; the id of a capture is not used again.
static thread_local unsigned long long t_capture_id = 0;
static thread_local cudaGraphNode_t t_capture_node = nullptr;

bool follows_linear(cudaStream_t s) {
    unsigned long long id = 0;
    cudaGraphNode_t node = nullptr;
    return capture_tail(s, &id, &node) && node == t_capture_node && id == t_capture_id;
}

void note_linear(cudaStream_t s) {
    if (!capture_tail(s, &t_capture_id, &t_capture_node)) t_capture_node = nullptr;
}

bool cluster_reduce_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("QF_CLUSTER_REDUCE");
        return !(e && e[0] == '0');
    }();
    return on;
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

// Which of the two kernels that read slab weights runs a linear called by itself. The streaming tcgen05 kernel takes its SMs whole
// and starts when its predecessor has ended, about 10 us a call that do not depend on the size; per byte it is faster, the more so
// the more rows. The GEMV kernel adds the partial sums of a row block's thread blocks one after the other, which are the more the
// longer K is. Measured on weights not in L2, calls back to back in a graph, GEMV's time / tcgen05's (blob in MiB):
//    rows  MiB   K 256   512  1024  2048  3072  4096  5120  6144  8192 14336
//    9     25    0.81  0.78  0.76  0.84  0.93  0.95  1.02  1.11  1.23  1.35
//          34    0.90  0.89  0.82  0.84  0.92  0.96  0.98  1.01  1.12  1.22
//          48    0.93  0.96  0.95  0.93  0.93  0.98  1.04  1.04  1.08  1.27
//          72    0.98  1.08  1.05  1.03  1.03  1.05  1.06  1.08  1.13  1.17
//    16    25    0.78  0.74  0.71  0.80  0.92  0.94  1.03  1.09  1.15  1.41
//          34    0.86  0.86  0.78  0.79  0.87  0.95  0.97  1.03  1.13  1.32
//          42    0.86  0.88  0.86  0.85  0.88  0.93  1.00  1.04  1.14  1.25
//          56    0.88  0.93  0.94  0.92  0.94  0.95  1.00  1.06  1.11  1.21
//          72    0.92  1.01  1.02  1.00  0.99  1.01  1.02  1.07  1.12  1.19
//          92    0.93  1.05  1.06  1.07  1.09  1.07  1.08  1.10  1.11  1.20
//    24    25    0.97  0.92  0.86  0.94  1.09  1.17  1.28  1.34  1.55  1.64
//          34    1.07  1.08  0.99  1.00  1.10  1.19  1.24  1.31  1.42  1.67
//    32    25    0.92  0.87  0.82  0.89  1.03  1.11  1.23  1.35  1.50  1.75
//          34    1.02  1.02  0.95  0.95  1.05  1.15  1.18  1.28  1.45  1.81
//          42    0.99  1.04  1.06  1.02  1.02  1.12  1.21  1.25  1.42  1.64
// In us: 9 rows 57344 x 8192 75.6 -> 57.6, 8192 x 28672 42.5 -> 33.6; 16 rows 83.2 -> 63.8 and 44.6 -> 35.0, 32 rows 135 -> 69.9 and
// 70.2 -> 38.7.
// Up to 8 rows the GEMV kernel serves whatever the size is: what the largest matrices gain waiting for each call is 1 % (4 rows,
// 57344 x 8192, SiLU * mul: 65.3 -> 64.7), and their sums would be made in another order than those of all smaller ones.
static bool stream_serves(const qf_linear_desc *d) {
    const int64_t mib = d->N / 64 * (d->K / 128) * QF_SLAB_UNIT_BYTES >> 20;
    if (d->M <= kSlabGemvRows) return false;
    if (d->M > 16) return mib >= (d->K >= 3072 ? 24 : d->M <= 24 ? 34 : 42);
    return d->K >= 512 && mib >= (d->K >= 8192 ? 24 : d->K >= 6144 ? 33 : d->K >= 5120 ? 42 : 72);
}

// Millions of codes from which the tcgen05 kernel is the faster one on canonical weights of N % 128 != 0 rows; -1: never. Its blocks take a
// tile of 128 rows and, up to 64 batch rows, an eighth of K at least; the GEMV kernel's take 64 rows, 8 batch rows and a piece of K that fills
// the device four times over. So this one loses where there are few tiles of long K, and on small matrices what its start-up and its sums cost.
// GEMV / tcgen05 kernel, times as fast, weights not in L2:
//   3, 4 rows    K 1024: N 10256 0.84, 12304 1.02    1536: 7184 0.95, 8208 1.05    2048: 5136 0.95, 6160 1.04    3072: 3088 0.99, 4112 1.02
//                4096: 2064 0.97, 3088 1.02, 4112 1.17    5120: 1552 0.94, 2064 1.01    with more than 8 splits: 4608: 1904 1.31
//                5504: 1296 1.37    6144: 1040 1.30    8192: 784 1.25    12416 to 14208: 0.87 to 1.22    14336: 784 to 2576 0.89 to 1.02, 3088 1.00
//                18944 to 28672: up to 2064 0.73 to 1.04 (16256: 592 1.11), 2960 and 3088 1.26
//   5 to 8       1024: 11840 0.79, 12304 1.11    1280: 9376 0.87, 10256 1.08    1536: 4112 0.93 to 0.99, 5136 1.00
//                2048: 3600 0.89 to 0.96, 4112 1.05    2560 to 16384: 0.93 and more    18944: 0.89 to 1.17 at 5
//                22784 to 28672: up to 1296 0.82 to 1.10 at 5 and 6, 0.88 to 1.19 at 8
//   9 to 16      up to 512: 0.95 and more but 128 x 57360 0.88    640: up to 18448 0.76 to 0.94, 20496 1.62
//                768: up to 8208 0.84 to 1.00, 12304 1.01, 18448 0.92    896: 7184, 8208 0.89 to 0.94, 10256 1.09
//                1152 to 1408: 3088, 4112 0.94 to 1.07    all else 1.0 to 3.7
//   17 to 64     128: 16400 0.80 to 0.85 up to 24    256: 8208 0.85 to 0.93 up to 40, 12304 0.95 and more    384, 512: 1.02 and more
//                640: up to 12304 0.80 to 0.93 up to 24, to 8208 0.89 to 0.93 at 32, to 7184 0.84 at 40
//                768, 896: up to 8208 0.87 to 1.09 up to 24, 3088 and 4112 0.75 to 0.91 to 64, 6160 1.12 from 32 on
//                1024: 2064, 2576 0.78 to 0.88 up to 24, then 0.99 and more but 2064 0.90 to 0.95 at 33 to 40
//                1152 to 1408: up to 3088 0.83 to 0.94 up to 24, to 2064 0.84 to 0.93 at 32, 1808 0.87 at 33 to 40    1536: 1552 0.95 and more
//                28672: 80 and 112 0.82 to 0.97 from 33 on, 144 0.85 to 0.92 up to 56 and 1.24 at 64, 208 0.91 up to 40 and 1.28 from 48 on
//   65 to 256    1024: 4112, 1536 and 1664: 3088 0.80 to 0.92 up to 72    2048: 2064 0.87 at 96 and 100
//                14336: 400 0.85 to 0.92 from 96 to 160    20480: 208 0.62 to 0.91 up to 200, 272 0.68 to 0.90 up to 160, then 1.05 and more
//                28672: 144 0.53 to 0.79, 208 0.60 to 0.78 up to 140, 272 0.73 to 0.97 up to 112, then 0.99 and more
//   more         1.5 and more
// (`on_chip`: the GEMV kernel has at most 8 splits, which a cluster sums.)
static double ragged_line(int64_t M, int64_t K, int64_t N, bool on_chip) {
    if (M <= 8) {
        if (K < 1024 || (M <= 4 && K > 14208 && N < 2688) || (M <= 6 && K > 20480 && N < 1536)) return -1;
        if (M > 4) return K < 1536 ? 12.5 : K < 2560 ? 8 : 6;
        return K < 1536 ? std::max<double>(12, 12288e-6 * K) : K < 2560 ? 12 : on_chip ? 10 : 6;
    }
    if (M <= 16) return K <= 512 || K >= 1024 ? 4 : K < 768 ? 12.5 : 9;
    if (M <= 64) {
        if (M > 32 && K > 16384 && N < (M > 56 ? 144 : M <= 40 && K >= 24576 ? 256 : 176)) return -1;
        if (K <= 512 || K >= 1536) return K < 384 && M <= (K < 256 ? 24 : 40) ? 2.5 : 2;
        if (K < 1024) return M <= 24 ? (K < 768 ? 9 : 7) : K >= 768 || M > 40 ? 4 : M <= 32 ? 6 : 5;
        return M <= 24 ? (K < 1280 ? 4 : 4.5) : M <= 32 ? (K < 1152 ? 2 : 2.95) : M <= 40 ? 2.4 : 2;
    }
    if (M <= 256 && (K > 16384 ? N < 176 || (N < 384 && M * N * K < 930000000) : K > 8192 && N < 512 && M * N < 65536)) return -1;
    if (M < 80 && K >= 1024 && K < 2048) return 5.2;
    if (M > 80 && M <= 104 && K > 1536 && K < 2560) return 4.5;
    return 4;
}

// Whether the tcgen05 kernel takes canonical weights of N % 128 != 0 rows, as the GEMV kernel can. Copies of scales and zeros are
// multiples of 16 bytes, also those of what is left for the last tile of 128 rows.
static bool gemm_serves_ragged(const qf_linear_desc *d) {
    if (d->weight_layout != QF_LAYOUT_CANONICAL || d->epilogue != QF_EPI_NONE || d->M < 3) return false;
    // A number of splits that the caller names is one of the GEMV kernel's, which runs them in shorter pieces where they are long (4 rows,
    // 14336 x 1040 in one split: 12.9 us there, 39.6 here).
    if (d->split_k != 0) return false;
    // What the GEMV kernel refuses stays refused, 32-bit and 16-bit results alike.
    qf_linear_desc other = *d;
    other.path = QF_PATH_GEMV;
    Plan gemv;
    if (make_plan(&other, &gemv, nullptr) != QF_OK) return false;
    if (d->zero_mode == QF_ZERO_U4 && d->N % 32 != 0) return false;
    // Sums of a whole split in one accumulator are 2e-7 to 4e-7 (of the outputs' rms) further off than the GEMV kernel's two accumulators
    // of shorter splits: 16-bit results, rounded by 1e-4 and more, do not show it; 32-bit ones keep that kernel.
    if (d->out_dtype == QF_F32) return false;
    const double line = ragged_line(d->M, d->K, d->N, gemv.split_k <= 8);
    return line >= 0 && d->K * d->N >= 1e6 * line;
}

int make_plan(const qf_linear_desc *d, Plan *p, std::string *why) {
    auto bad = [&](int st, const char *m) {
        if (why) *why = m;
        return st;
    };
    if (!d) return bad(QF_ERR_BAD_ARG, "desc is null");
    if (d->M < 0 || d->N <= 0 || d->K <= 0) return bad(QF_ERR_BAD_ARG, "M, N, K must be positive (M may be 0)");
    if (d->K % 128 != 0) return bad(QF_ERR_BAD_ARG, "K must be a multiple of 128");
    if (d->N % 16 != 0) return bad(QF_ERR_BAD_ARG, "N must be a multiple of 16");
    if (d->group_size <= 0 || d->group_size % 128 != 0 || d->K % d->group_size != 0)
        return bad(QF_ERR_UNSUPPORTED, "group_size must be a multiple of 128 that divides K");
    if (d->act_dtype != QF_F16 && d->act_dtype != QF_BF16)
        return bad(QF_ERR_UNSUPPORTED, "act_dtype must be QF_F16 or QF_BF16");
    if (d->out_dtype != QF_F16 && d->out_dtype != QF_BF16 && d->out_dtype != QF_F32)
        return bad(QF_ERR_UNSUPPORTED, "out_dtype must be QF_F16, QF_BF16 or QF_F32");
    if (d->zero_mode != QF_ZERO_CONST && d->zero_mode != QF_ZERO_U4 && d->zero_mode != QF_ZERO_I8)
        return bad(QF_ERR_BAD_ARG, "unknown zero_mode");
    if (d->zero_mode == QF_ZERO_CONST && (d->zero_const < -128 || d->zero_const > 127))
        return bad(QF_ERR_BAD_ARG, "zero_const must fit a signed 8-bit zero point");
    if (d->split_k < 0) return bad(QF_ERR_BAD_ARG, "split_k must be >= 0");
    if (d->weight_layout != QF_LAYOUT_CANONICAL && d->weight_layout != QF_LAYOUT_INTERLEAVED &&
        d->weight_layout != QF_LAYOUT_TILED && d->weight_layout != QF_LAYOUT_GEMV_SLAB)
        return bad(QF_ERR_BAD_ARG, "unknown weight_layout");
    if (d->epilogue != QF_EPI_NONE && d->epilogue != QF_EPI_SILU_MUL && d->epilogue != QF_EPI_RESIDUAL_ADD)
        return bad(QF_ERR_BAD_ARG, "unknown epilogue");
    for (int i = 0; i < 3; ++i)
        if (d->reserved[i] != 0) return bad(QF_ERR_BAD_ARG, "reserved fields must be zero");
    p->slab = false;
    p->stream = false;
    p->pair = false;
    if (d->weight_layout == QF_LAYOUT_GEMV_SLAB) {
        if (d->path == QF_PATH_GEMM)
            return bad(QF_ERR_BAD_ARG, "QF_LAYOUT_GEMV_SLAB weights are read by the GEMV path only");
        if (d->N % 64 != 0) return bad(QF_ERR_BAD_ARG, "QF_LAYOUT_GEMV_SLAB needs N to be a multiple of 64");
        if (d->M > QF_SLAB_MAX_M)
            return bad(QF_ERR_UNSUPPORTED, "QF_LAYOUT_GEMV_SLAB serves M <= 32; use a tcgen05 layout for larger batches");
        if (d->split_k == 0 && d->path == QF_PATH_AUTO && stream_serves(d)) {
            p->stream = true;
            p->path = QF_PATH_GEMV;
            p->split_k = 2 * kSmCount;
            p->chunks_per_split = 0;
            p->m_tiles = 1;
            p->bn = d->M <= 16 ? 16 : 32;
            p->ws_partial_bytes = stream_workspace_bytes(d->M);
            p->ws_counter_bytes = kCounterBytes;
            return QF_OK;
        }
        int grid = 1, depth = 1;
        slab_geometry(d->M, d->N, d->K, kSmCount, d->split_k, &grid, &depth);
        p->slab = true;
        p->path = QF_PATH_GEMV;
        p->split_k = grid;
        p->chunks_per_split = depth;
        p->m_tiles = 1;
        p->bn = 8 * ((slab_m_pad(d->M) + 7) / 8);
        p->ws_partial_bytes = slab_workspace_bytes(grid, d->M);
        p->ws_counter_bytes = 0;
        return QF_OK;
    }

    int path = d->path;
    if (path == QF_PATH_AUTO) {
        // M <= 2: the GEMV kernel wins on small matrices (short start-up, 4 blocks per SM); on large ones the tcgen05
        // kernel streams faster (measured at M=1: 42 MB 24.4 vs 17.7 us, 59 MB 33.0 vs 22.0 us, 117 MB 56.5 vs
        // 36.5 us with prepacked weights; 19.8 / 24.7 / 41.7 us with canonical ones; a tie around 32 MB).
        const int64_t wbytes = d->K * d->N / 2;
        const bool big = d->N % 128 == 0 &&
                         wbytes >= (d->weight_layout == QF_LAYOUT_CANONICAL ? (int64_t)40 << 20 : (int64_t)32 << 20);
        path = (d->M <= 2 && !big) ? QF_PATH_GEMV : QF_PATH_GEMM;
    }
    if (path != QF_PATH_GEMV && path != QF_PATH_GEMM) return bad(QF_ERR_BAD_ARG, "unknown path");
    if (d->epilogue != QF_EPI_NONE) {
        // the fused epilogues live in the streaming GEMV kernel (above) and in the tcgen05 kernel
        if (d->path == QF_PATH_GEMV || d->N % 128 != 0)
            return bad(QF_ERR_UNSUPPORTED,
                       "a fused epilogue needs QF_LAYOUT_GEMV_SLAB weights or the tcgen05 path (N % 128 == 0)");
        path = QF_PATH_GEMM;
    }
    // Any multiple of 16 rows of weights where the kernel may be chosen: the last tile of 128 is cut short (gemm_serves_ragged)
    if (path == QF_PATH_GEMM && d->N % 128 != 0 && !(d->path == QF_PATH_AUTO && gemm_serves_ragged(d))) {
        if (d->path == QF_PATH_GEMM) return bad(QF_ERR_BAD_ARG, "the GEMM path needs N to be a multiple of 128");
        path = QF_PATH_GEMV;
    }
    if (path == QF_PATH_GEMV && d->weight_layout != QF_LAYOUT_CANONICAL) {
        if (d->N % 128 != 0) return bad(QF_ERR_UNSUPPORTED, "interleaved weights need N to be a multiple of 128");
        path = QF_PATH_GEMM;  // only the tcgen05 kernel reads the interleaved layout
    }
    p->path = path;
    const int chunks = (int)(d->K / 128);
    if (path == QF_PATH_GEMV) {
        p->m_tiles = (int)((d->M + 7) / 8);
        if (p->m_tiles < 1) p->m_tiles = 1;
        p->bn = 8;
        const int64_t col_blocks = (d->N + 63) / 64;
        int split;
        if (d->split_k > 0) {
            split = d->split_k;
        } else {
            const int64_t base = col_blocks * p->m_tiles;
            const int64_t target = (int64_t)kSmCount * 4;
            split = (int)((target + base / 2) / base);
            const int max_split = chunks / 4 > 0 ? chunks / 4 : 1;
            if (split > max_split) split = max_split;
            if (split < 1) split = 1;
        }
        if (split > chunks) split = chunks;
        if (d->split_k == 0 && split > 8 && split <= 10 && chunks % 8 == 0 && chunks / 8 <= 32)
            split = 8;  // an even split that fits one thread-block cluster (on-chip reduction)
        int cps = (chunks + split - 1) / split;
        if (cps > 32) cps = 32;
        split = (chunks + cps - 1) / cps;
        p->split_k = split;
        p->chunks_per_split = cps;
        if (col_blocks * p->m_tiles > kMaxCounters) split = 1, cps = chunks > 32 ? 32 : chunks;
        if (cps * split < chunks) return bad(QF_ERR_UNSUPPORTED, "K too large for this N on the GEMV path");
        p->split_k = split;
        p->chunks_per_split = cps;
        if (split > 1) {
            p->ws_partial_bytes = (size_t)split * p->m_tiles * 8 * d->N * sizeof(float);
            p->ws_counter_bytes = kCounterBytes;
        } else {
            p->ws_partial_bytes = 0;
            p->ws_counter_bytes = 0;
        }
    } else {
        // As few batch tiles as a width of 256 allows, all of one width: the smallest multiple of 16 that covers M. (Tiles
        // of 16, 32, 64, 128 or 256 rows ran M = 777 as 1024 rows; 777 x 4096 x 4096 f16, canonical: 38.5 -> 35.1 us.)
        p->m_tiles = d->M > 256 ? (int)((d->M + 255) / 256) : 1;
        const int64_t rows = d->M > p->m_tiles ? (d->M + p->m_tiles - 1) / p->m_tiles : 1;
        const int64_t tiles = (int64_t)p->m_tiles * ((d->N + 127) / 128);
        auto width = [&](int step) { return (int)((rows + step - 1) / step * step); };
        // Splits of K for batch tiles of bn rows in k-blocks of bk codes, and k-blocks per split.
        auto splits = [&](int bn, int bk, int *kbps_out) {
            const int kblocks = (int)(d->K / bk);
            int split;
            if (d->split_k > 0) {
                split = d->split_k;
            } else {
                const int64_t slots = (int64_t)kSmCount * (bn <= 64 ? 2 : 1);  // two narrow CTAs fit one SM
                split = (int)(slots / tiles);
                if (split < 1) split = 1;
                // narrow tiles: at most 8 splits, the size of a portable thread-block cluster; 8 splits summed on chip
                // beat 16 or 32 summed through global memory (measured, 8 tiles, K = 8192: 9.3 -> 6.9 us at M = 16,
                // 17.7 -> 9.6 us at M = 64)
                if (bn <= 64 && split > 8) split = 8;
            }
            if (split > kblocks) split = kblocks;
            int kbps = (kblocks + split - 1) / split;
            // at least 512 codes a block (with 256, K = 4096, N = 1024 took 38.7 us instead of 30.3 at M = 256)
            const int min_kbps = d->split_k > 0 ? 1 : std::min(kblocks, 512 / bk);
            if (kbps < min_kbps) kbps = min_kbps;
            split = (kblocks + kbps - 1) / kbps;
            if (d->split_k == 0 && split > 2 && kblocks % split != 0) {
                // a slightly smaller split that divides K evenly beats an uneven one: fewer partial tiles to write and
                // sum and no short last split (measured on K = 14336: 8 x 14 k-blocks is 3-7 % faster than 8 x 13 + 8)
                for (int s2 = split - 1; s2 >= split - 2 && s2 >= 2; --s2)
                    if (kblocks % s2 == 0 && (kblocks / s2) * 20 <= kbps * 23) {
                        split = s2;
                        kbps = kblocks / s2;
                        break;
                    }
            }
            if (d->split_k == 0 && bn <= 64 && split >= 2 && split <= 8 && tiles * split > kClusterMaxBlocks &&
                kClusterMaxBlocks / tiles >= 2) {
                // A launch of more than kClusterMaxBlocks blocks cannot run as one wave of thread-block clusters and
                // would sum its partial tiles through global memory; fewer, longer splits that keep the on-chip
                // reduction are faster (measured, 48 tiles: 6 splits 10.0 / 15.8 us at M = 16 / 64, 5 splits 9.1 / 11.9).
                split = (int)(kClusterMaxBlocks / tiles);
                kbps = (kblocks + split - 1) / split;
                split = (kblocks + kbps - 1) / kbps;
            }
            if (tiles > kMaxCounters) split = 1, kbps = kblocks;
            *kbps_out = kbps;
            return split;
        };
        // Above 64 rows two neighbouring weight tiles can share one batch tile, whose width is then a multiple of 32. The start
        // and end of a pair cost about a microsecond, and what it gives back grows with the codes a block runs through (K over
        // the split) and depends on the width: up to 128 rows either form works on 128 codes at a time and a pair only loads
        // less of X; above, a block alone works on 64, which tells most where the MMAs of 64 codes are short. Measured for
        // M 72 to 1462, N 1024 to 28672, K 1536 to 28672, pair against alone, mean over the shapes of each range of codes:
        //   width     512     1024    1536    2048    3072    4096    6144    8192    more
        //   <= 128   -5.4 %  -6.8   -12.6    -3.8    -7.2    +0.7    -4.2    +4.0    +8.6
        //   <= 192   -2.1    -0.4    +0.5    +7.4   +12.0   +14.8   +17.3   +20.3   +19.8
        //   wider    -2.2    -1.8    -5.5    -1.3    +1.2    +2.6    +4.8    +7.1    +7.3
        int kbps = 1, split = 1;
        p->pair = false;
        if (rows > 64 && d->N % 256 == 0) {
            split = splits(width(32), gemm_block_k(width(32), true), &kbps);
            const int64_t codes = (int64_t)kbps * gemm_block_k(width(32), true);
            // (1536 codes at widths up to 192: 3 to 8 % gained, but 6 to 25 % lost where they are all of K and N = 14336)
            p->pair = d->K >= 2048 && codes >= (width(32) <= 128 ? 7168 : width(32) <= 192 ? 1536 : 2176);
        }
        const int bn = width(p->pair ? 32 : 16);
        if (!p->pair) split = splits(bn, gemm_block_k(bn, false), &kbps);
        p->bn = bn;
        p->split_k = split;
        p->chunks_per_split = kbps;
        if (split > 1) {
            p->ws_partial_bytes = (size_t)split * p->m_tiles * bn * d->N * sizeof(float);
            p->ws_counter_bytes = kCounterBytes;
        } else {
            p->ws_partial_bytes = 0;
            p->ws_counter_bytes = 0;
        }
    }
    return QF_OK;
}

static int check_linear_args(qf_ctx *ctx, const qf_linear_desc *d, const void *X, const void *qw, const void *scales,
                             const void *zeros, const void *Y) {
    if (d->weight_layout == QF_LAYOUT_GEMV_SLAB) {
        // the blob carries scales and zeros
        if (!X || !qw || !Y) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
        if (!aligned16(X) || !aligned16(qw) || !aligned16(Y))
            return fail(ctx, QF_ERR_BAD_ARG, "device pointers must be 16-byte aligned");
        return QF_OK;
    }
    if (!X || !qw || !scales || !Y) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (d->zero_mode != QF_ZERO_CONST && !zeros) return fail(ctx, QF_ERR_BAD_ARG, "zero_mode needs a qzeros tensor");
    if (d->zero_mode == QF_ZERO_U4 && d->N % 8 != 0) return fail(ctx, QF_ERR_BAD_ARG, "QF_ZERO_U4 needs N % 8 == 0");
    if (!aligned16(X) || !aligned16(qw) || !aligned16(scales) || !aligned16(Y) || (zeros && !aligned16(zeros)))
        return fail(ctx, QF_ERR_BAD_ARG, "device pointers must be 16-byte aligned");
    return QF_OK;
}

// A plan that the GEMV kernel can step in for (gemm_serves_ragged).
static bool ragged_gemm(const qf_linear_desc *d, const Plan &plan) { return plan.path == QF_PATH_GEMM && d->N % 128 != 0; }

// Everything that a linear's launch relies on, and its plan. M == 0 needs no tensors. Without a context: all but the current device.
static int check_linear(qf_ctx *ctx, const qf_linear_desc *desc, const void *X, const void *qweight, const void *scales,
                        const void *qzeros_or_null, const void *Y, const void *residual, const void *workspace,
                        size_t workspace_bytes, Plan *plan) {
    std::string why;
    int st = make_plan(desc, plan, &why);
    if (st != QF_OK) return fail(ctx, st, why);
    if (desc->M == 0) return QF_OK;
    st = check_linear_args(ctx, desc, X, qweight, scales, qzeros_or_null, Y);
    if (st != QF_OK) return st;
    if (ctx) st = check_current_device(ctx);
    if (st != QF_OK) return st;
    if (desc->epilogue == QF_EPI_RESIDUAL_ADD && (!residual || !aligned16(residual)))
        return fail(ctx, QF_ERR_BAD_ARG, "QF_EPI_RESIDUAL_ADD needs a 16-byte aligned residual tensor");
    if (desc->epilogue == QF_EPI_SILU_MUL && desc->N % 16 != 0)
        return fail(ctx, QF_ERR_BAD_ARG, "QF_EPI_SILU_MUL needs N (gate and up rows together) to be a multiple of 16");
    size_t need = plan->ws_partial_bytes + plan->ws_counter_bytes;
    if (ragged_gemm(desc, *plan) && need > 0 && (!workspace || workspace_bytes < need)) {
        // what the GEMV kernel can do with its own scratch (none, where it does not split) is its
        qf_linear_desc d = *desc;
        d.path = QF_PATH_GEMV;
        if ((st = make_plan(&d, plan, &why)) != QF_OK) return fail(ctx, st, why);
        need = plan->ws_partial_bytes + plan->ws_counter_bytes;
    }
    if (need > 0) {
        if (!workspace || workspace_bytes < need)
            return fail(ctx, QF_ERR_WORKSPACE, "workspace smaller than qf_w4a16_workspace_bytes(desc)");
        if (!aligned16(workspace)) return fail(ctx, QF_ERR_BAD_ARG, "workspace must be 16-byte aligned");
    }
    return QF_OK;
}

// Slab weights, and nothing in the descriptor that names a kernel.
static bool slab_any(const qf_linear_desc *d) {
    return d->weight_layout == QF_LAYOUT_GEMV_SLAB && d->split_k == 0 && d->path == QF_PATH_AUTO;
}

// Linears that qf_w4a16_linear_batched runs as one launch. (One without rows goes alone: it has no launch, and its pointers were not
// looked at.)
static bool chains(const qf_linear_desc *d) {
    return d->M > 0 && slab_any(d) && d->N > 0 && d->N % 64 == 0 && d->K > 0 && d->K % 128 == 0 && (d->M <= kSlabGemvRows ? slab_chain_takes(d) : d->N % 128 == 0);
}
// The workspace of that launch.
static size_t chain_workspace_bytes(int64_t M) {
    return kCounterBytes + (M <= kSlabGemvRows ? slab_chain_workspace_bytes() : stream_workspace_bytes(M));
}

// Slots of partial sums of a chain of more than kSlabGemvRows rows in this workspace.
static int chain_slots(int64_t M, size_t workspace_bytes) {
    return workspace_bytes >= kCounterBytes + stream_workspace_bytes(M, kChainSlots) ? kChainSlots : kStreamSlots;
}

// How many of the linears from entry i on one launch could take, those linears, and whether it does or they go one by one. (A linear
// with which something is wrong goes alone, and its check says what. They are checked once it is known that a chain would pay: most
// batches that go one by one are checked there.)
static int chain_from(qf_ctx *ctx, int i, int count, const qf_linear_desc *descs, const void *const *X, const void *const *qweight,
                      void *const *Y, const void *const *residual, const void *workspace, size_t workspace_bytes,
                      std::vector<StreamLinear> *run, bool *pays) {
    run->clear();
    const bool gemv = descs[i].M <= kSlabGemvRows;
    Plan plan;
    for (int j = i; j < count && j - i < kStreamMaxLinears && chains(&descs[j]) && descs[j].M == descs[i].M; ++j) {
        run->push_back(StreamLinear{&descs[j], X[j], qweight[j], residual ? residual[j] : nullptr, Y[j], 1, 0});
        if (gemv) continue;
        // K is cut as the tcgen05 kernel cuts it for the same sizes in its own layouts: the sums are the same bits
        qf_linear_desc d = descs[j];
        d.weight_layout = QF_LAYOUT_INTERLEAVED;
        if (make_plan(&d, &plan, nullptr) != QF_OK || plan.path != QF_PATH_GEMM) {
            run->pop_back();
            break;
        }
        run->back().split = plan.split_k;
        run->back().per = plan.chunks_per_split;
    }
    int n = run->size() > 1 ? stream_chain_length(run->data(), (int)run->size()) : 1;
    const auto faster = [&] {
        return n > 1 && workspace_bytes >= chain_workspace_bytes(descs[i].M) &&
               (gemv ? slab_chain_pays : stream_chain_pays)(run->data(), n);
    };
    *pays = faster();
    for (int k = 0; *pays && k < n; ++k) {
        const StreamLinear &x = (*run)[k];
        if (check_linear(ctx, x.d, x.X, x.blob, nullptr, nullptr, x.Y, x.residual, workspace, workspace_bytes, &plan) != QF_OK) {
            n = k;
            *pays = faster();
            break;
        }
    }
    return std::max(n, 1);
}

static int launch_linear(qf_ctx *ctx, const qf_linear_desc *desc, const Plan &plan, const void *X, const void *qweight,
                         const void *scales, const void *qzeros_or_null, void *Y, const void *residual, void *workspace,
                         cudaStream_t s) {
    if (plan.slab) return launch_gemv_slab(ctx, desc, plan, X, qweight, Y, residual, workspace, s);
    if (plan.stream) {
        const int st = launch_stream(ctx, StreamLinear{desc, X, qweight, residual, Y, 1, 0}, workspace, kCounterBytes, s);
        if (st != kStreamNoRoom) return st;
        qf_linear_desc d = *desc;
        d.path = QF_PATH_GEMV;
        Plan other;  // its workspace is the smaller one
        if (make_plan(&d, &other, nullptr) != QF_OK) return fail(ctx, QF_ERR_UNSUPPORTED, "no kernel for this linear");
        return launch_gemv_slab(ctx, desc, other, X, qweight, Y, residual, workspace, s);
    }
    if (plan.path == QF_PATH_GEMV) return launch_gemv(ctx, desc, plan, X, qweight, scales, qzeros_or_null, Y, workspace, s);
    return launch_gemm(ctx, desc, plan, X, qweight, scales, qzeros_or_null, Y, residual, workspace, s);
}

}  // namespace qf

using namespace qf;

extern "C" {

int qf_version(void) { return QF_RT_VERSION; }

const char *qf_status_string(int status) {
    switch (status) {
        case QF_OK: return "QF_OK";
        case QF_ERR_BAD_ARG: return "QF_ERR_BAD_ARG";
        case QF_ERR_UNSUPPORTED: return "QF_ERR_UNSUPPORTED";
        case QF_ERR_CUDA: return "QF_ERR_CUDA";
        case QF_ERR_NCCL: return "QF_ERR_NCCL";
        case QF_ERR_TIMEOUT: return "QF_ERR_TIMEOUT";
        case QF_ERR_UNIMPLEMENTED: return "QF_ERR_UNIMPLEMENTED";
        case QF_ERR_WORKSPACE: return "QF_ERR_WORKSPACE";
        default: return "QF_ERR_UNKNOWN";
    }
}

int qf_ctx_create(qf_ctx **out, int device) {
    if (!out) return QF_ERR_BAD_ARG;
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0) return QF_ERR_CUDA;  // no CPU fallback exists
    if (device < 0 || device >= count) return QF_ERR_BAD_ARG;
    DeviceGuard guard(device);  // the caller's current device is restored on every return path
    if (!guard.ok()) return QF_ERR_CUDA;
    qf_ctx *ctx = new (std::nothrow) qf_ctx();
    if (!ctx) return QF_ERR_CUDA;
    ctx->device = device;
    int major = 0;
    if (cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess) {
        delete ctx;
        return QF_ERR_CUDA;
    }
    if (major != 10) {
        delete ctx;
        return QF_ERR_UNSUPPORTED;  // built for sm_100a only
    }
    int st = gemv_init(ctx);
    if (st == QF_OK) st = gemm_init(ctx);
    if (st == QF_OK) st = gemv_slab_init(ctx);
    if (st == QF_OK) st = stream_init(ctx);
    if (st == QF_OK) st = slab_chain_init(ctx);
    if (st != QF_OK) {
        delete ctx;
        return st;
    }
    *out = ctx;
    return QF_OK;
}

int qf_ctx_destroy(qf_ctx *ctx) {
    if (!ctx) return QF_OK;
    DeviceGuard guard(ctx->device);
    cudaDeviceSynchronize();
    for (auto &sl : ctx->host_slot) {
        if (sl.x) cudaFree(sl.x);
        if (sl.y) cudaFree(sl.y);
        if (sl.copied_in) cudaEventDestroy(sl.copied_in);
        if (sl.kernel_done) cudaEventDestroy(sl.kernel_done);
    }
    if (ctx->mapped_x) cudaFree(ctx->mapped_x);
    for (void *q : ctx->retired) cudaFree(q);
    if (ctx->order) cudaEventDestroy(ctx->order);
    if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
    if (ctx->host_status) cudaFreeHost(ctx->host_status);
    delete ctx;
    return QF_OK;
}

const char *qf_last_error(const qf_ctx *ctx) { return ctx ? ctx->last_error.c_str() : "null context"; }

int qf_unpack_int4(qf_ctx *ctx, const void *packed_i8, void *out_i8, int64_t rows, int64_t packed_cols, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (rows < 0 || packed_cols < 0) return fail(ctx, QF_ERR_BAD_ARG, "negative extent");
    if (rows == 0 || packed_cols == 0) return QF_OK;
    if (!packed_i8 || !out_i8) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (((uintptr_t)out_i8 & 1u) != 0) return fail(ctx, QF_ERR_BAD_ARG, "output must be 2-byte aligned");
    return launch_unpack(ctx, packed_i8, out_i8, rows, packed_cols, (cudaStream_t)stream);
}

int qf_pack_int4(qf_ctx *ctx, const void *codes_i8, void *out_i8, int64_t n_bytes, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (n_bytes < 0) return fail(ctx, QF_ERR_BAD_ARG, "negative extent");
    if (n_bytes == 0) return QF_OK;
    if (!codes_i8 || !out_i8) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (!aligned16(codes_i8) || ((uintptr_t)out_i8 & 7u))
        return fail(ctx, QF_ERR_BAD_ARG, "codes must be 16-byte and the output 8-byte aligned");
    int st = check_current_device(ctx);
    if (st != QF_OK) return st;
    return launch_pack(ctx, codes_i8, out_i8, n_bytes, (cudaStream_t)stream);
}

int qf_quantize_w4(qf_ctx *ctx, const void *weight, int dtype, int64_t N, int64_t K, int group_size, int symmetric,
                   void *codes_i8, void *scales, int scale_dtype, void *zeros_i8_or_null, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (N <= 0 || K <= 0 || group_size <= 0 || group_size % 4 != 0 || K % group_size != 0 || K > INT32_MAX)
        return fail(ctx, QF_ERR_BAD_ARG, "group_size must be a multiple of 4 that divides K");
    if (N * (K / group_size) > INT32_MAX) return fail(ctx, QF_ERR_BAD_ARG, "too many groups");
    if (dtype != QF_F16 && dtype != QF_BF16 && dtype != QF_F32) return fail(ctx, QF_ERR_UNSUPPORTED, "unknown weight type");
    if (scale_dtype != QF_F16 && scale_dtype != QF_BF16)
        return fail(ctx, QF_ERR_UNSUPPORTED, "scales are QF_F16 or QF_BF16");
    if (!weight || !codes_i8 || !scales || (!symmetric && !zeros_i8_or_null))
        return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (!aligned16(weight) || !aligned16(codes_i8)) return fail(ctx, QF_ERR_BAD_ARG, "device pointers must be 16-byte aligned");
    int st = check_current_device(ctx);
    if (st != QF_OK) return st;
    return launch_quantize(ctx, weight, dtype, N, K, group_size, symmetric != 0, codes_i8, scales, scale_dtype,
                           zeros_i8_or_null, (cudaStream_t)stream);
}

int qf_dequant_w4(qf_ctx *ctx, const qf_linear_desc *desc, const void *qweight, const void *scales,
                  const void *qzeros_or_null, void *w_out, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (!desc) return fail(ctx, QF_ERR_BAD_ARG, "desc is null");
    if (desc->weight_layout != QF_LAYOUT_CANONICAL)
        return fail(ctx, QF_ERR_UNSUPPORTED, "qf_dequant_w4 reads canonical weights only (undo the prepack first)");
    qf_linear_desc d = *desc;
    d.M = 1;
    d.path = QF_PATH_GEMV;
    d.out_dtype = d.act_dtype;
    d.epilogue = QF_EPI_NONE;
    Plan plan;
    std::string why;
    int st = make_plan(&d, &plan, &why);
    if (st != QF_OK) return fail(ctx, st, why);
    st = check_linear_args(ctx, &d, w_out, qweight, scales, qzeros_or_null, w_out);
    if (st != QF_OK) return st;
    return launch_dequant(ctx, &d, qweight, scales, qzeros_or_null, w_out, (cudaStream_t)stream);
}

size_t qf_w4a16_workspace_bytes(const qf_linear_desc *desc) {
    Plan plan;
    if (make_plan(desc, &plan, nullptr) != QF_OK) return 0;
    size_t need = plan.ws_partial_bytes + plan.ws_counter_bytes;
    if (ragged_gemm(desc, plan)) {  // an exchanging call takes the GEMV kernel
        qf_linear_desc d = *desc;
        d.path = QF_PATH_GEMV;
        if (make_plan(&d, &plan, nullptr) == QF_OK) need = std::max(need, plan.ws_partial_bytes + plan.ws_counter_bytes);
    }
    if (desc->weight_layout == QF_LAYOUT_GEMV_SLAB && desc->split_k == 0) {
        // An exchanging call on the same descriptor may divide the weights among more thread blocks. That is also what the
        // streaming GEMV kernel needs where it steps in for the tcgen05 kernel.
        const int64_t units = desc->N / 64 * (desc->K / 128);
        need = std::max(need, slab_workspace_bytes((int)std::min<int64_t>(units, slab_exchange_grid(desc, kSmCount)), desc->M));
    }
    return need;
}

size_t qf_w4a16_batched_workspace_bytes(int count, const qf_linear_desc *descs) {
    size_t need = 0;
    int64_t slots = 0;  // of partial sums, of the linears since one that does not go with the one before
    for (int i = 0; descs && i < count; ++i) {
        need = std::max(need, qf_w4a16_workspace_bytes(&descs[i]));
        const bool run = i > 0 && chains(&descs[i]) && chains(&descs[i - 1]) && descs[i].M == descs[i - 1].M &&
                         descs[i].act_dtype == descs[i - 1].act_dtype;
        if (run) need = std::max(need, chain_workspace_bytes(descs[i].M));
        if (!run) slots = 0;
        if (descs[i].M <= kSlabGemvRows || !chains(&descs[i])) continue;
        qf_linear_desc d = descs[i];
        d.weight_layout = QF_LAYOUT_INTERLEAVED;
        Plan plan;
        if (make_plan(&d, &plan, nullptr) == QF_OK && plan.split_k > 1) slots += row_blocks(d) * plan.split_k;
        if (run && slots > kStreamSlots) need = std::max(need, kCounterBytes + stream_workspace_bytes(d.M, kChainSlots));
    }
    return need;
}

int qf_w4a16_plan(const qf_linear_desc *desc, int32_t *path_out, int32_t *split_k_out) {
    Plan plan;
    int st = make_plan(desc, &plan, nullptr);
    if (st != QF_OK) return st;
    if (path_out) *path_out = plan.path;
    if (split_k_out) *split_k_out = plan.split_k;
    return QF_OK;
}

int qf_w4a16_linear_fused(qf_ctx *ctx, const qf_linear_desc *desc, const void *X, const void *qweight,
                          const void *scales, const void *qzeros_or_null, void *Y, const void *residual,
                          void *workspace, size_t workspace_bytes, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    Plan plan;
    const int st = check_linear(ctx, desc, X, qweight, scales, qzeros_or_null, Y, residual, workspace, workspace_bytes, &plan);
    if (st != QF_OK || desc->M == 0) return st;
    return launch_linear(ctx, desc, plan, X, qweight, scales, qzeros_or_null, Y, residual, workspace, (cudaStream_t)stream);
}

int qf_w4a16_linear(qf_ctx *ctx, const qf_linear_desc *desc, const void *X, const void *qweight, const void *scales,
                    const void *qzeros_or_null, void *Y, void *workspace, size_t workspace_bytes, void *stream) {
    if (desc && desc->epilogue == QF_EPI_RESIDUAL_ADD)
        return fail(ctx, QF_ERR_BAD_ARG, "QF_EPI_RESIDUAL_ADD takes its residual through qf_w4a16_linear_fused");
    return qf_w4a16_linear_fused(ctx, desc, X, qweight, scales, qzeros_or_null, Y, nullptr, workspace, workspace_bytes,
                                 stream);
}

int qf_w4a16_linear_batched(qf_ctx *ctx, int count, const qf_linear_desc *descs, const void *const *X,
                            const void *const *qweight, const void *const *scales, const void *const *qzeros,
                            void *const *Y, const void *const *residual, void *workspace, size_t workspace_bytes,
                            void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (count < 0) return fail(ctx, QF_ERR_BAD_ARG, "negative count");
    if (count == 0) return QF_OK;
    if (!descs || !X || !qweight || !Y) return fail(ctx, QF_ERR_BAD_ARG, "null argument array");
    std::vector<StreamLinear> run;
    for (int i = 0, alone = 0; i < count; ++i) {
        bool pays = false;
        const int n = i < alone ? 1 : chain_from(ctx, i, count, descs, X, qweight, Y, residual, workspace, workspace_bytes, &run, &pays);
        alone = std::max(alone, i + n);
        if (pays) {
            const int64_t M = descs[i].M;
            const int st = M <= kSlabGemvRows ? launch_slab_chain(ctx, run.data(), n, workspace, kCounterBytes, (cudaStream_t)stream)
                                              : launch_stream_chain(ctx, run.data(), n, workspace, kCounterBytes,
                                                                    chain_slots(M, workspace_bytes), (cudaStream_t)stream);
            if (st != QF_OK && st != kStreamNoRoom) return st;
            if (st == QF_OK) {
                i += n - 1;
                continue;
            }
        }
        const int st = qf_w4a16_linear_fused(ctx, &descs[i], X[i], qweight[i], scales ? scales[i] : nullptr,
                                             qzeros ? qzeros[i] : nullptr, Y[i], residual ? residual[i] : nullptr,
                                             workspace, workspace_bytes, stream);
        if (st != QF_OK) {
            ctx->last_error = "entry " + std::to_string(i) + ": " + ctx->last_error;
            return st;
        }
    }
    return QF_OK;
}

int qf_w4a16_batched_launches(qf_ctx *ctx, int count, const qf_linear_desc *descs, const void *const *X, const void *const *qweight,
                              void *const *Y, const void *const *residual, const void *workspace, size_t workspace_bytes) {
    if (!ctx || count < 0 || (count > 0 && (!descs || !X || !qweight || !Y))) return -1;
    std::vector<StreamLinear> run;
    int launches = 0;
    for (int i = 0, n; i < count; i += n) {
        bool pays = false;
        n = chain_from(ctx, i, count, descs, X, qweight, Y, residual, workspace, workspace_bytes, &run, &pays);
        if (pays) ++launches;
        else
            for (int j = i; j < i + n; ++j) launches += descs[j].M > 0;
    }
    return launches;
}

int qf_w4a16_batched_plan(int count, const qf_linear_desc *descs, const void *const *X, const void *const *qweight, void *const *Y,
                          const void *const *residual, const void *workspace, size_t workspace_bytes, int32_t *out) {
    if (count < 0 || (count > 0 && (!descs || !X || !qweight || !Y || !out))) return QF_ERR_BAD_ARG;
    std::vector<StreamLinear> run;
    ChainPlan plan;
    for (int i = 0, n, launch = 0; i < count; i += n) {
        bool pays = false;
        n = chain_from(nullptr, i, count, descs, X, qweight, Y, residual, workspace, workspace_bytes, &run, &pays);
        int32_t *o = out + (size_t)i * QF_BATCHED_PLAN_WORDS;
        std::fill(o, o + (size_t)n * QF_BATCHED_PLAN_WORDS, -1);
        const bool gemv = descs[i].M <= kSlabGemvRows;
        if (!pays || (gemv && !plan_slab_chain(run.data(), n, kSmCount, &plan))) {
            for (int j = 0; j < n; ++j)
                if (descs[i + j].M > 0) o[j * QF_BATCHED_PLAN_WORDS] = launch++;
            continue;
        }
        if (!gemv) plan_stream_chain(run.data(), n, 2 * kSmCount, chain_slots(descs[i].M, workspace_bytes), &plan);
        for (size_t q = 0; q < plan.phases.size(); ++q) {
            const ChainPhase &c = plan.phases[q];
            for (int k = c.first; k < c.first + c.count; ++k) {
                const ChainLinear &x = plan.linears[plan.order[k]];
                const int32_t words[QF_BATCHED_PLAN_WORDS] = {launch, (int32_t)q, c.wait[0], c.wait[1], x.slot, x.slots,
                                                              gemv ? kSlabChainPlaces * x.first_sm + x.home : c.slots_wait, gemv ? x.grid : -1};
                std::copy(words, words + QF_BATCHED_PLAN_WORDS, o + (size_t)plan.order[k] * QF_BATCHED_PLAN_WORDS);
            }
        }
        ++launch;
    }
    return QF_OK;
}

size_t qf_prepack_bytes(int layout, int64_t N, int64_t K) {
    if (N <= 0 || K <= 0 || K % 128 != 0) return 0;
    switch (layout) {
        case QF_LAYOUT_CANONICAL: return (size_t)N * (size_t)K / 2;
        case QF_LAYOUT_INTERLEAVED:
        case QF_LAYOUT_TILED: return N % 128 == 0 ? (size_t)N * (size_t)K / 2 : 0;
        case QF_LAYOUT_GEMV_SLAB: return N % 64 == 0 ? (size_t)(N / 64) * (size_t)(K / 128) * QF_SLAB_UNIT_BYTES : 0;
        default: return 0;
    }
}

int qf_prepack_gemv_slab(qf_ctx *ctx, const qf_linear_desc *desc, const void *qweight, const void *scales,
                         const void *qzeros_or_null, void *blob_out, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (!desc) return fail(ctx, QF_ERR_BAD_ARG, "desc is null");
    qf_linear_desc d = *desc;
    d.M = 1;
    d.path = QF_PATH_AUTO;
    d.weight_layout = QF_LAYOUT_GEMV_SLAB;
    d.epilogue = QF_EPI_NONE;
    d.out_dtype = d.act_dtype;
    Plan plan;
    std::string why;
    int st = make_plan(&d, &plan, &why);
    if (st != QF_OK) return fail(ctx, st, why);
    if (!qweight || !scales || !blob_out) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (d.zero_mode != QF_ZERO_CONST && !qzeros_or_null) return fail(ctx, QF_ERR_BAD_ARG, "zero_mode needs a qzeros tensor");
    if (!aligned16(qweight) || !aligned16(scales) || !aligned16(blob_out) || (qzeros_or_null && !aligned16(qzeros_or_null)))
        return fail(ctx, QF_ERR_BAD_ARG, "device pointers must be 16-byte aligned");
    if (blob_out == qweight) return fail(ctx, QF_ERR_BAD_ARG, "the blob must not alias the canonical weights");
    st = check_current_device(ctx);
    if (st != QF_OK) return st;
    return launch_slab_prepack(ctx, &d, qweight, scales, qzeros_or_null, blob_out, (cudaStream_t)stream);
}

int qf_unpack_gemv_slab(qf_ctx *ctx, int64_t N, int64_t K, const void *blob, void *qweight_out, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (N <= 0 || K <= 0 || N % 64 != 0 || K % 128 != 0)
        return fail(ctx, QF_ERR_BAD_ARG, "QF_LAYOUT_GEMV_SLAB needs N % 64 == 0 and K % 128 == 0");
    if (!blob || !qweight_out) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (!aligned16(blob) || !aligned16(qweight_out)) return fail(ctx, QF_ERR_BAD_ARG, "device pointers must be 16-byte aligned");
    int st = check_current_device(ctx);
    if (st != QF_OK) return st;
    return launch_slab_unpack(ctx, N, K, blob, qweight_out, (cudaStream_t)stream);
}

int qf_repack_kn_to_canonical(qf_ctx *ctx, const void *w_kn, int packed_along_n, int64_t K, int64_t N,
                              void *qweight_out, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (K <= 0 || N <= 0 || K % 8 != 0 || N % 2 != 0)
        return fail(ctx, QF_ERR_BAD_ARG, "qf_repack_kn_to_canonical needs K % 8 == 0 and N % 2 == 0");
    if (!w_kn || !qweight_out) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (w_kn == qweight_out) return fail(ctx, QF_ERR_BAD_ARG, "in and out must not alias");
    if (((uintptr_t)qweight_out & 3u) != 0) return fail(ctx, QF_ERR_BAD_ARG, "output must be 4-byte aligned");
    int st = check_current_device(ctx);
    if (st != QF_OK) return st;
    return launch_repack_kn(ctx, w_kn, packed_along_n ? 1 : 0, K, N, qweight_out, (cudaStream_t)stream);
}

int qf_w4a16_gemv_static_scratch(qf_ctx *ctx, const qf_linear_desc *desc, const void *X, const void *qweight,
                                 const void *scales, const void *qzeros_or_null, void *Y, void *stream) {
    if (!desc) return fail(ctx, QF_ERR_BAD_ARG, "desc is null");
    qf_linear_desc d = *desc;
    d.path = QF_PATH_GEMV;
    if (d.weight_layout != QF_LAYOUT_CANONICAL)
        return fail(ctx, QF_ERR_UNSUPPORTED, "the GEMV kernel reads canonical weights only");
    Plan plan;
    std::string why;
    int st = make_plan(&d, &plan, &why);
    if (st != QF_OK) return fail(ctx, st, why);
    if (d.M == 0) return QF_OK;
    if (!X || !qweight || !scales || !Y) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (d.zero_mode != QF_ZERO_CONST && !qzeros_or_null) return fail(ctx, QF_ERR_BAD_ARG, "zero_mode needs a qzeros tensor");
    if (!aligned16(X) || !aligned16(qweight) || !aligned16(scales) || !aligned16(Y) ||
        (qzeros_or_null && !aligned16(qzeros_or_null)))
        return fail(ctx, QF_ERR_BAD_ARG, "device pointers must be 16-byte aligned");
    return launch_gemv_static(ctx, &d, plan, X, qweight, scales, qzeros_or_null, Y, (cudaStream_t)stream);
}

// Page-locked host buffers up to these sizes: a kernel of the caller's stream fetches the activations and the linear writes its
// result to the host, two launches one behind the other instead of two copies, a second stream and three events. The copy
// engine moves larger ones, on a stream of its own. Measured on weights not in L2, waiting for each call / calls back to back,
// copied -> fetched:
//   2 rows 4096 -> 14336 (16 and 57 KB)       48.3 -> 40.3 us / 36.1 -> 24.3
//   64 rows 512 -> 512 (64 and 64 KB)         35.0 -> 25.0    / 17.2 -> 10.2
//   16 rows 4096 -> 4112 fp32 (128, 257 KB)   49.1 -> 38.5    / 27.6 -> 19.9  (GEMV kernel: four bytes a thread)
//   64 rows 4096 -> 14336 (0.5 and 1.8 MB)    87.0 -> 75.6    / 68.5 -> 49.9
//   256 rows 4096 -> 4096 (2 and 2 MB)         135 -> 113     / 89.6 -> 80.8
//   64 rows 14336 -> 4096 (1.8 and 0.5 MB)    85.9 -> 77.0    / 56.4 -> 57.7
//   73 rows 14336 -> 512 (2 and 0.07 MB)      90.9 -> 81.8    / 46.4 -> 57.1  (long K, small result: the one loss seen below 2 MB)
//   128 rows 4096 -> 14336 (1 and 3.7 MB)      155 -> 128     /  100 -> 114
// The tcgen05 kernel without a split stores fp32 results as half sectors, 32 bytes a thread in two pieces, which PCIe takes at
// 15 GB/s; these go to the host up to 192 KB:
//   64 rows 512 -> 512 fp32 (64 and 128 KB)   35.0 -> 30.0    / 23.0 -> 15.0
//   128 rows 512 -> 512 fp32 (128, 256 KB)    43.0 -> 45.5    / 23.2 -> 25.2
//   1000 rows 512 -> 512 fp32 (1 and 2 MB)    93.2 -> 180     / 62.3 -> 156
constexpr size_t kMappedX = 2u << 20, kMappedY = 2u << 20, kMappedHalfSectors = 192u << 10;

// Staging buffers only grow; the outgrown one is retired, not freed (see qf_ctx::HostSlot).
static int grow(qf_ctx *ctx, void **buf, size_t *have, size_t need) {
    if (*have >= need) return QF_OK;
    if (*buf) ctx->retired.push_back(*buf);
    *buf = nullptr;
    *have = 0;
    size_t cap = (need + ((size_t)1 << 20) - 1) & ~(((size_t)1 << 20) - 1);
    QF_CUDA_TRY(ctx, cudaMalloc(buf, cap));
    *have = cap;
    return QF_OK;
}

// The address under which kernels reach [p, p + bytes), if all of it is one range of page-locked host memory; else null.
static void *mapped_host(const void *p, size_t bytes) {
    typedef CUresult (*AttributesFn)(unsigned, CUpointer_attribute *, void **, CUdeviceptr);
    static const AttributesFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        const bool ok = cudaGetDriverEntryPoint("cuPointerGetAttributes", &f, cudaEnableDefault, &r) == cudaSuccess &&
                        r == cudaDriverEntryPointSuccess;
        return ok ? (AttributesFn)f : (AttributesFn) nullptr;
    }();
    if (!fn || !aligned16(p)) return nullptr;
    unsigned type = 0;
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[4] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                   CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void *to[4] = {&type, &dev, &start, &size};
    if (fn(4, what, to, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS || type != CU_MEMORYTYPE_HOST || dev == 0) return nullptr;
    if (dev < start || dev - start > size || size - (size_t)(dev - start) < bytes) return nullptr;
    return (void *)(uintptr_t)dev;
}

// Puts the copy stream behind all that `s` holds so far: no result is pending for its copies any more.
static int order_copies(qf_ctx *ctx, cudaStream_t s) {
    if (ctx->copy_stream) {
        QF_CUDA_TRY(ctx, cudaEventRecord(ctx->order, s));
        QF_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->order, 0));
    }
    ctx->n_pending = 0;
    return QF_OK;
}

static bool pending(const qf_ctx *ctx, const qf_ctx::HostRange &x) {
    for (int i = 0; i < ctx->n_pending; ++i)
        if (x.meets(ctx->pending_y[i])) return true;
    return false;
}

// After a call has been enqueued; one that waits leaves nothing pending.
static int note_result(qf_ctx *ctx, const qf_ctx::HostRange &y, bool waits, cudaStream_t s) {
    ctx->last_y = waits ? qf_ctx::HostRange{0, 0} : y;
    if (waits) return QF_OK;
    for (int i = 0; i < ctx->n_pending; ++i)
        if (ctx->pending_y[i].begin <= y.begin && y.end <= ctx->pending_y[i].end) return QF_OK;
    if (ctx->n_pending == qf_ctx::kMaxPending) {
        const int st = order_copies(ctx, s);
        if (st != QF_OK) return st;
    }
    ctx->pending_y[ctx->n_pending++] = y;
    return QF_OK;
}

static int enqueue_host_linear(qf_ctx *ctx, const qf_linear_desc *desc, const void *X_host, const void *qweight,
                               const void *scales, const void *qzeros_or_null, void *Y_host, void *workspace,
                               size_t workspace_bytes, void *stream, bool waits) {
    if (!ctx) return QF_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(ctx->host_mutex);
    if (!desc) return fail(ctx, QF_ERR_BAD_ARG, "desc is null");
    if (!X_host || !Y_host) return fail(ctx, QF_ERR_BAD_ARG, "null host pointer");
    if (desc->M == 0) return QF_OK;
    if (desc->epilogue == QF_EPI_RESIDUAL_ADD)
        return fail(ctx, QF_ERR_BAD_ARG, "QF_EPI_RESIDUAL_ADD takes its residual through qf_w4a16_linear_fused");
    // Everything is checked before anything is allocated or enqueued. The linear's X and Y will be staging buffers or mapped
    // addresses, aligned like this one.
    alignas(16) static const char aligned[16] = {};
    Plan plan;
    int st = check_linear(ctx, desc, aligned, qweight, scales, qzeros_or_null, aligned, nullptr, workspace, workspace_bytes, &plan);
    if (st != QF_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) cudaGetLastError();  // the launch says what is wrong with the stream
    if (capture != cudaStreamCaptureStatusNone)
        return fail(ctx, QF_ERR_UNSUPPORTED, "linears on host buffers cannot be captured");
    const size_t xb = (size_t)desc->M * desc->K * 2;
    const int64_t out_cols = desc->epilogue == QF_EPI_SILU_MUL ? desc->N / 2 : desc->N;
    const size_t yb = (size_t)desc->M * out_cols * (desc->out_dtype == QF_F32 ? 4 : 2);
    const qf_ctx::HostRange x_range = {(uintptr_t)X_host, (uintptr_t)X_host + xb}, y_range = {(uintptr_t)Y_host, (uintptr_t)Y_host + yb};
    void *x = nullptr, *y = nullptr;
    const bool half_sectors = plan.path == QF_PATH_GEMM && plan.split_k == 1 && desc->out_dtype == QF_F32;
    if (xb <= kMappedX && yb <= (half_sectors ? kMappedHalfSectors : kMappedY) &&
        (x = mapped_host(X_host, xb)) != nullptr && (y = mapped_host(Y_host, yb)) != nullptr) {
        if (!ctx->mapped_x) QF_CUDA_TRY(ctx, cudaMalloc(&ctx->mapped_x, kMappedX));
        st = launch_fetch(ctx, x, ctx->mapped_x, (int64_t)xb, x_range.meets(ctx->last_y), s);
        if (st != QF_OK) return st;
        st = launch_linear(ctx, desc, plan, ctx->mapped_x, qweight, scales, qzeros_or_null, y, nullptr, workspace, s);
        return st != QF_OK ? st : note_result(ctx, y_range, waits, s);
    }
    const bool first = !ctx->copy_stream;
    if (first) {
        QF_CUDA_TRY(ctx, cudaEventCreateWithFlags(&ctx->order, cudaEventDisableTiming));
        QF_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
        for (auto &sl : ctx->host_slot) {
            QF_CUDA_TRY(ctx, cudaEventCreateWithFlags(&sl.copied_in, cudaEventDisableTiming));
            QF_CUDA_TRY(ctx, cudaEventCreateWithFlags(&sl.kernel_done, cudaEventDisableTiming));
        }
    }
    if (first || pending(ctx, x_range)) {
        st = order_copies(ctx, s);
        if (st != QF_OK) return st;
    }
    qf_ctx::HostSlot &sl = ctx->host_slot[ctx->host_next];
    ctx->host_next ^= 1;
    st = grow(ctx, &sl.x, &sl.x_bytes, xb);
    if (st != QF_OK) return st;
    st = grow(ctx, &sl.y, &sl.y_bytes, yb);
    if (st != QF_OK) return st;
    // activations: on the copy stream, as soon as the slot's previous kernel (two calls ago) has read its own
    QF_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->copy_stream, sl.kernel_done, 0));  // no-op before the first record
    QF_CUDA_TRY(ctx, cudaMemcpyAsync(sl.x, X_host, xb, cudaMemcpyHostToDevice, ctx->copy_stream));
    QF_CUDA_TRY(ctx, cudaEventRecord(sl.copied_in, ctx->copy_stream));
    QF_CUDA_TRY(ctx, cudaStreamWaitEvent(s, sl.copied_in, 0));
    st = launch_linear(ctx, desc, plan, sl.x, qweight, scales, qzeros_or_null, sl.y, nullptr, workspace, s);
    if (st != QF_OK) return st;
    QF_CUDA_TRY(ctx, cudaEventRecord(sl.kernel_done, s));
    // the result goes back on the caller's stream: synchronising it is all the caller has to do
    QF_CUDA_TRY(ctx, cudaMemcpyAsync(Y_host, sl.y, yb, cudaMemcpyDeviceToHost, s));
    return note_result(ctx, y_range, waits, s);
}

int qf_w4a16_linear_host_async(qf_ctx *ctx, const qf_linear_desc *desc, const void *X_host, const void *qweight,
                         const void *scales, const void *qzeros_or_null, void *Y_host, void *workspace,
                         size_t workspace_bytes, void *stream) {
    return enqueue_host_linear(ctx, desc, X_host, qweight, scales, qzeros_or_null, Y_host, workspace, workspace_bytes, stream,
                               false);
}

int qf_w4a16_linear_host(qf_ctx *ctx, const qf_linear_desc *desc, const void *X_host, const void *qweight,
                         const void *scales, const void *qzeros_or_null, void *Y_host, void *workspace,
                         size_t workspace_bytes, void *stream) {
    const int st = enqueue_host_linear(ctx, desc, X_host, qweight, scales, qzeros_or_null, Y_host, workspace, workspace_bytes,
                                       stream, true);
    if (st != QF_OK) return st;
    QF_CUDA_TRY(ctx, cudaStreamSynchronize((cudaStream_t)stream));
    return QF_OK;
}

int qf_prepack_w4(qf_ctx *ctx, const void *qweight_in, void *qweight_out, int64_t n_words, int to_canonical,
                  void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (n_words < 0) return fail(ctx, QF_ERR_BAD_ARG, "negative extent");
    if (n_words == 0) return QF_OK;
    if (!qweight_in || !qweight_out) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (((uintptr_t)qweight_in & 3u) || ((uintptr_t)qweight_out & 3u))
        return fail(ctx, QF_ERR_BAD_ARG, "weights must be 4-byte aligned");
    return launch_prepack(ctx, qweight_in, qweight_out, n_words, to_canonical, (cudaStream_t)stream);
}

int qf_prepack_w4_tiled(qf_ctx *ctx, const void *qweight_in, void *qweight_out, int64_t N, int64_t K,
                        int to_canonical, void *stream) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (N <= 0 || K <= 0 || N % 128 != 0 || K % 128 != 0)
        return fail(ctx, QF_ERR_BAD_ARG, "the tiled layout needs N and K to be multiples of 128");
    if (!qweight_in || !qweight_out) return fail(ctx, QF_ERR_BAD_ARG, "null tensor pointer");
    if (qweight_in == qweight_out) return fail(ctx, QF_ERR_BAD_ARG, "in and out must not alias");
    if (((uintptr_t)qweight_in & 15u) || ((uintptr_t)qweight_out & 15u))
        return fail(ctx, QF_ERR_BAD_ARG, "weights must be 16-byte aligned");
    return launch_prepack_tiled(ctx, qweight_in, qweight_out, N, K, to_canonical, (cudaStream_t)stream);
}

int qf_ctx_status(const qf_ctx *ctx) {
    if (!ctx) return QF_ERR_BAD_ARG;
    return ctx->host_status ? *(volatile int *)ctx->host_status : QF_OK;
}

int qf_ctx_clear_status(qf_ctx *ctx) {
    if (!ctx) return QF_ERR_BAD_ARG;
    if (ctx->host_status) *(volatile int *)ctx->host_status = QF_OK;
    return QF_OK;
}

int64_t qf_launch_count(void) { return (int64_t)g_launch_count.load(); }

}  // extern "C"
