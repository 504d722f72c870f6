// K1: qf.unpack as a stand-alone kernel, its inverse, and the materialising qf.dequant(qf.unpack(w)).
//
// All are streaming kernels bound by HBM: unpack reads 1 byte and writes 2 per input byte, pack the other way round;
// dequant reads 0.5 byte and writes 2 per weight.
#include "qf_common.cuh"

namespace qf {

__device__ __forceinline__ uint4 ld_stream16(const void *p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_stream8(const void *p) {
    uint2 v;
    asm volatile("ld.global.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
// 32 bytes with one store instruction (a whole sector per thread): 32-byte aligned addresses only.
__device__ __forceinline__ void st_stream32(void *p, const uint4 &a, const uint4 &b) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                 "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// 4 packed bytes -> 8 output bytes.  lo = low nibbles, hi = high nibbles (one per byte lane);
// prmt interleaves them: (lo.b0, hi.b0, lo.b1, hi.b1) and (lo.b2, hi.b2, lo.b3, hi.b3).
__device__ __forceinline__ void unpack_word(uint32_t w, uint32_t &o0, uint32_t &o1) {
    const uint32_t lo = w & 0x0f0f0f0fu;
    const uint32_t hi = (w >> 4) & 0x0f0f0f0fu;
    o0 = prmt(lo, hi, 0x5140u);
    o1 = prmt(lo, hi, 0x7362u);
}

// 16 input bytes per step, four steps in flight per thread, one 32-byte store each. Where the output is only aligned to 16 bytes (WIDE is
// false) the sectors lie across two threads: each stores its second half with the first half of the thread behind it (64 MB in 31.7 us; two
// stores of 16 bytes a thread, half a sector each, 41.3 to 49.9; aligned 32.7, a byte per thread 57.2). The up to 15 bytes behind the last
// whole step are unpacked by the first threads of block 0.
// Four loads per thread before the first store, and whole-sector stores, are what the memory system needs: one load and
// two 16-byte stores 32 bytes apart ran at 4.5 TB/s (28672 x 4096 bytes in 77.4 us).
constexpr int UNPACK_STEPS = 4;
template <bool WIDE>
__global__ void __launch_bounds__(256) unpack_vec_kernel(const uint8_t *in, uint8_t *out,
                                                         int64_t n_vec, int tail) {
    griddep_begin();
    const int64_t first = (int64_t)blockIdx.x * (256 * UNPACK_STEPS) + threadIdx.x;
    uint4 v[UNPACK_STEPS];
#pragma unroll
    for (int j = 0; j < UNPACK_STEPS; ++j)
        v[j] = first + j * 256 < n_vec ? ld_stream16(in + (first + j * 256) * 16) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int j = 0; j < UNPACK_STEPS; ++j) {
        if (WIDE && first + j * 256 >= n_vec) continue;
        uint4 a, b;
        unpack_word(v[j].x, a.x, a.y);
        unpack_word(v[j].y, a.z, a.w);
        unpack_word(v[j].z, b.x, b.y);
        unpack_word(v[j].w, b.z, b.w);
        uint8_t *dst = out + (first + j * 256) * 32;
        if (WIDE) {
            st_stream32(dst, a, b);
        } else {
            const int lane = threadIdx.x & 31;
            const uint4 next = make_uint4(__shfl_down_sync(0xffffffffu, a.x, 1), __shfl_down_sync(0xffffffffu, a.y, 1),
                                          __shfl_down_sync(0xffffffffu, a.z, 1), __shfl_down_sync(0xffffffffu, a.w, 1));
            if (first + j * 256 >= n_vec) continue;
            if (lane == 0) *reinterpret_cast<uint4 *>(dst) = a;
            if (lane < 31 && first + j * 256 + 1 < n_vec) st_stream32(dst + 16, b, next);
            else *reinterpret_cast<uint4 *>(dst + 16) = b;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < tail) {
        const int64_t i = n_vec * 16 + threadIdx.x;
        const uint8_t byte = in[i];
        out[2 * i] = byte & 0x0f;
        out[2 * i + 1] = byte >> 4;
    }
}

// Any alignment (of the output: 2): one byte per thread and step. The pointers may alias as far as the compiler knows, so it
// moves no load ahead of a store: the loads of LOOP_STEPS steps are written ahead of their stores, without a condition but in the
// last pass (58.7 MB at an odd address: 49.6 us, with a condition in every pass 54.5, one step at a time 105.4).
constexpr int LOOP_STEPS = 4;
__global__ void __launch_bounds__(256) unpack_byte_kernel(const uint8_t *in, uint8_t *out,
                                                          int64_t n_bytes) {
    griddep_begin();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + (LOOP_STEPS - 1) * stride < n_bytes; i += LOOP_STEPS * stride) {
        uint8_t b[LOOP_STEPS];
#pragma unroll
        for (int j = 0; j < LOOP_STEPS; ++j) b[j] = in[i + j * stride];
#pragma unroll
        for (int j = 0; j < LOOP_STEPS; ++j) {
            uchar2 o;
            o.x = b[j] & 0x0f;
            o.y = b[j] >> 4;
            reinterpret_cast<uchar2 *>(out)[i + j * stride] = o;
        }
    }
    uint8_t b[LOOP_STEPS];
#pragma unroll
    for (int j = 0; j < LOOP_STEPS; ++j)
        if (i + j * stride < n_bytes) b[j] = in[i + j * stride];
#pragma unroll
    for (int j = 0; j < LOOP_STEPS; ++j) {
        if (i + j * stride >= n_bytes) break;
        uchar2 o;
        o.x = b[j] & 0x0f;
        o.y = b[j] >> 4;
        reinterpret_cast<uchar2 *>(out)[i + j * stride] = o;
    }
}

int launch_unpack(qf_ctx *ctx, const void *packed, void *out, int64_t rows, int64_t packed_cols, cudaStream_t s) {
    const int64_t n_bytes = rows * packed_cols;
    if (n_bytes == 0) return QF_OK;
    cudaError_t e;
    if ((uintptr_t)packed % 16 == 0 && (uintptr_t)out % 16 == 0) {
        const int64_t n_vec = n_bytes / 16;
        int64_t blocks = (n_vec + 256 * UNPACK_STEPS - 1) / (256 * UNPACK_STEPS);
        if (blocks < 1) blocks = 1;
        auto *fn = (uintptr_t)out % 32 == 0 ? unpack_vec_kernel<true> : unpack_vec_kernel<false>;
        e = launch_kernel(fn, dim3((unsigned)blocks), dim3(256), 0, s, pdl_enabled(), (const uint8_t *)packed, (uint8_t *)out, n_vec,
                          (int)(n_bytes % 16));
    } else {
        int64_t blocks = (n_bytes + 255) / 256;
        if (blocks > (int64_t)ctx->sm_count * 16) blocks = (int64_t)ctx->sm_count * 16;
        e = launch_kernel(unpack_byte_kernel, dim3((unsigned)blocks), dim3(256), 0, s, pdl_enabled(), (const uint8_t *)packed,
                          (uint8_t *)out, n_bytes);
    }
    return launched(ctx, e, "unpack");
}

// Mapped host memory to device memory, 16 bytes per thread. Bound by the round trip over PCIe for a few rows of activations, then
// by its bandwidth. The source is the caller's and final when the call is made, so its way begins before earlier work of the stream
// has ended; the destination is written behind the wait. (14336 -> 4096, 8 rows, calls back to back: 17.4 us; 30.7 with the read
// behind the wait.) Where it is the result of an earlier call (`behind`), the linear that writes it may be running: read behind the wait.
__global__ void __launch_bounds__(256) fetch_kernel(const uint4 *src, uint4 *dst, int64_t n_vec, int behind) {
    griddep_launch_dependents();
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (behind) griddep_wait();
    if (i < n_vec) v = ld_stream16(src + i);
    if (!behind) griddep_wait();
    if (i < n_vec) dst[i] = v;
}

int launch_fetch(qf_ctx *ctx, const void *src, void *dst, int64_t bytes, bool behind, cudaStream_t s) {
    const int64_t n_vec = bytes / 16;
    return launched(ctx, launch_kernel(fetch_kernel, dim3((unsigned)((n_vec + 255) / 256)), dim3(256), 0, s, pdl_enabled(),
                                       (const uint4 *)src, (uint4 *)dst, n_vec, behind ? 1 : 0),
                    "fetch");
}

// The inverse: out[i] = (codes[2i] & 15) | (codes[2i + 1] & 15) << 4. 16 codes in, 8 bytes out per step.
__device__ __forceinline__ uint32_t pack_words(uint32_t lo, uint32_t hi) {
    // each word: bytes c0 c1 c2 c3 -> (c0 | c1 << 4) in byte 0, (c2 | c3 << 4) in byte 2
    lo &= 0x0f0f0f0fu;
    hi &= 0x0f0f0f0fu;
    return prmt(lo | (lo >> 4), hi | (hi >> 4), 0x6420u);
}
__global__ void __launch_bounds__(256) pack_vec_kernel(const uint8_t *codes, uint8_t *out,
                                                       int64_t n_vec, int tail) {
    griddep_begin();
    const int64_t first = (int64_t)blockIdx.x * (256 * UNPACK_STEPS) + threadIdx.x;
    uint4 v[UNPACK_STEPS];
#pragma unroll
    for (int j = 0; j < UNPACK_STEPS; ++j)
        if (first + j * 256 < n_vec) v[j] = ld_stream16(codes + (first + j * 256) * 16);
#pragma unroll
    for (int j = 0; j < UNPACK_STEPS; ++j)
        if (first + j * 256 < n_vec)
            reinterpret_cast<uint2 *>(out)[first + j * 256] = make_uint2(pack_words(v[j].x, v[j].y), pack_words(v[j].z, v[j].w));
    if (blockIdx.x == 0 && threadIdx.x < tail) {
        const int64_t i = n_vec * 8 + threadIdx.x;
        out[i] = (uint8_t)((codes[2 * i] & 0x0f) | (codes[2 * i + 1] & 0x0f) << 4);
    }
}

int launch_pack(qf_ctx *ctx, const void *codes, void *out, int64_t n_bytes, cudaStream_t s) {
    const int64_t n_vec = n_bytes / 8;
    int64_t blocks = (n_vec + 256 * UNPACK_STEPS - 1) / (256 * UNPACK_STEPS);
    if (blocks < 1) blocks = 1;
    return launched(ctx, launch_kernel(pack_vec_kernel, dim3((unsigned)blocks), dim3(256), 0, s, pdl_enabled(), (const uint8_t *)codes,
                                       (uint8_t *)out, n_vec, (int)(n_bytes % 8)),
                    "pack");
}

// Nibble permutation inside each word: qf_prepack_w4, in place or not (a thread writes only words that it has read). Loads ahead
// of the stores as in unpack_byte_kernel: 28672 x 8192 42.3 us, with a condition in every pass 45.9, one step at a time 66.5.
__global__ void __launch_bounds__(256) prepack_kernel(const uint32_t *in, uint32_t *out,
                                                      int64_t n_words, int to_canonical) {
    griddep_begin();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + (LOOP_STEPS - 1) * stride < n_words; i += LOOP_STEPS * stride) {
        uint32_t w[LOOP_STEPS];
#pragma unroll
        for (int j = 0; j < LOOP_STEPS; ++j) w[j] = in[i + j * stride];
#pragma unroll
        for (int j = 0; j < LOOP_STEPS; ++j) out[i + j * stride] = to_canonical ? deinterleave_word(w[j]) : interleave_word(w[j]);
    }
    uint32_t w[LOOP_STEPS];
#pragma unroll
    for (int j = 0; j < LOOP_STEPS; ++j)
        if (i + j * stride < n_words) w[j] = in[i + j * stride];
#pragma unroll
    for (int j = 0; j < LOOP_STEPS; ++j)
        if (i + j * stride < n_words) out[i + j * stride] = to_canonical ? deinterleave_word(w[j]) : interleave_word(w[j]);
}

int launch_prepack(qf_ctx *ctx, const void *in, void *out, int64_t n_words, int to_canonical, cudaStream_t s) {
    int64_t blocks = (n_words + 255) / 256;
    if (blocks > (int64_t)ctx->sm_count * 16) blocks = (int64_t)ctx->sm_count * 16;
    return launched(ctx, launch_kernel(prepack_kernel, dim3((unsigned)blocks), dim3(256), 0, s, pdl_enabled(), (const uint32_t *)in,
                                       (uint32_t *)out, n_words, to_canonical),
                    "prepack");
}

// canonical word (n, j) <-> tiled word ((nt * KB + kb) * 128 + r) * 16 + w, n = nt*128 + r, j = kb*16 + w.
// A block moves one tile (8 KB, contiguous on the tiled side): two 16-byte pieces per thread, four threads to the 64
// bytes of a row.
__global__ void __launch_bounds__(256) prepack_tiled_kernel(const uint4 *in, uint4 *out,
                                                            int KB, int to_canonical) {
    griddep_begin();
    const int nt = (int)(blockIdx.x / (unsigned)KB), kb = (int)(blockIdx.x % (unsigned)KB);
    const int64_t tile = (int64_t)blockIdx.x * 512;
    const int64_t canon0 = ((int64_t)nt * 128 * KB + kb) * 4;
    int64_t canon[2];
    uint4 piece[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = h * 256 + (int)threadIdx.x;
        canon[h] = canon0 + (int64_t)(i >> 2) * KB * 4 + (i & 3);
        piece[h] = in[to_canonical ? tile + i : canon[h]];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = h * 256 + (int)threadIdx.x;
        uint4 v = piece[h];
        if (to_canonical)
            v = make_uint4(deinterleave_word(v.x), deinterleave_word(v.y), deinterleave_word(v.z), deinterleave_word(v.w));
        else
            v = make_uint4(interleave_word(v.x), interleave_word(v.y), interleave_word(v.z), interleave_word(v.w));
        out[to_canonical ? canon[h] : tile + i] = v;
    }
}

int launch_prepack_tiled(qf_ctx *ctx, const void *in, void *out, int64_t N, int64_t K, int to_canonical,
                         cudaStream_t s) {
    const int64_t tiles = (N / 128) * (K / 128);
    if (tiles > INT32_MAX) return fail(ctx, QF_ERR_UNSUPPORTED, "matrix too large");
    return launched(ctx, launch_kernel(prepack_tiled_kernel, dim3((unsigned)tiles), dim3(256), 0, s, pdl_enabled(), (const uint4 *)in,
                                       (uint4 *)out, (int)(K / 128), to_canonical),
                    "tiled prepack");
}

// W[K, N] (one code per byte, or two per byte along N) -> canonical qweight [N, K/8] words. One thread per output
// word; consecutive threads take consecutive n, so the reads are coalesced (the 4-byte writes are not: one-time op).
__global__ void __launch_bounds__(256) repack_kn_kernel(const uint8_t *w_kn, int packed_along_n,
                                                        int64_t K, int64_t N, uint32_t *out) {
    griddep_begin();
    const int64_t words_per_row = K >> 3;
    const int64_t total = N * words_per_row;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int64_t n = i % N;
        const int64_t j = i / N;
        uint32_t word = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int64_t k = 8 * j + c;
            uint32_t code;
            if (packed_along_n) {
                const uint32_t b = w_kn[k * (N >> 1) + (n >> 1)];
                code = (n & 1) ? (b >> 4) & 0xFu : b & 0xFu;
            } else {
                code = w_kn[k * N + n] & 0xFu;
            }
            word |= code << (4 * c);
        }
        out[n * words_per_row + j] = word;
    }
}

int launch_repack_kn(qf_ctx *ctx, const void *w_kn, int packed_along_n, int64_t K, int64_t N, void *out,
                     cudaStream_t s) {
    const int64_t total = N * (K / 8);
    int64_t blocks = (total + 255) / 256;
    if (blocks > (int64_t)ctx->sm_count * 16) blocks = (int64_t)ctx->sm_count * 16;
    return launched(ctx, launch_kernel(repack_kn_kernel, dim3((unsigned)blocks), dim3(256), 0, s, pdl_enabled(), (const uint8_t *)w_kn,
                                       packed_along_n, K, N, (uint32_t *)out),
                    "repack");
}

// A block converts 16 rows x 512 codes: a warp covers 512 codes of a row, a thread two neighbouring words of it (8 bytes
// in, one 32-byte store out), in two rows (four where those are short), all loads in flight. The words of a thread lie in one quantisation group, so
// there is one scale and one zero per row; neighbouring rows' scales share sectors, which the block's rows find in L1.
// One word per thread with a 64-bit division to find its row ran at 3.2 TB/s (14336 x 4096 bf16 in 45.6 us).
// Grid: blocks of columns in x, so that those that run together write whole rows, blocks of rows in y and, where there are more than 65535 of
// them, in z. (Blocks of 32 rows, one below the other: 14336 x 4096 bf16 25.1 us instead of 23.9, 28672 x 8192 95.1 instead of 88.4, all bytes at
// the copy rate 22.6 and 90; 32 rows in the present order 24.3 and 88.9, 64 rows 27.6 and 97.3.)
// Rows of one or two groups leave most of a block's threads idle, and many of them are bound by the blocks' starts and ends: they go 32 to
// a block, four to a thread (16 -> 32 rows a block, f16: 65536 x 128, constant zero 8.01 -> 6.92 us, 262144 x 256 33.3 -> 30.7, 262144 x 128 with
// packed zeros 32.0 -> 29.6; but 4096 x 128 1.89 -> 2.19, 262144 x 256 with packed zeros 34.9 -> 36.8, 32768 x 384 5.63 -> 6.04, and with 8-bit zeros
// 524288 x 128 62.0 -> 64.6).
static int dequant_rows(int zmode, int64_t N, int64_t K) {
    if (zmode == QF_ZERO_CONST) return K <= 256 && N >= 32768 ? 4 : 2;
    return zmode == QF_ZERO_U4 && K <= 128 && N >= 65536 ? 4 : 2;
}
template <bool BF16, int ZMODE, bool WIDE, int ROWS>
__global__ void __launch_bounds__(256) dequant_kernel(const uint32_t *qw,
                                                      const uint16_t *scales,
                                                      const void *zeros, int zero_const,
                                                      uint4 *w_out, int64_t N, int words_per_row,
                                                      int group_words) {
    griddep_begin();
    const int64_t j = (int64_t)blockIdx.x * 64 + (threadIdx.x & 31) * 2;
    if (j >= words_per_row) return;
    const int64_t n0 = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * (8 * ROWS) + (threadIdx.x >> 5);
    const int64_t gi = (int)j / group_words;
    uint2 w[ROWS];
    ZeroScale<BF16> zs[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        if (n0 + 8 * r < N) w[r] = ld_stream8(qw + (n0 + 8 * r) * words_per_row + j);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int64_t n = n0 + 8 * r;
        if (n < N) zs[r].set(load_zero<ZMODE>(zeros, zero_const, gi, n, N), scales[gi * N + n]);
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int64_t n = n0 + 8 * r;
        if (n >= N) continue;
        uint4 o[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t p[4];
            dequant8<BF16>(h ? w[r].y : w[r].x, zs[r], p);
            // p[i] = (c_i, c_{i+4}) -> memory order (c0,c1)(c2,c3)(c4,c5)(c6,c7)
            o[h] = make_uint4(prmt(p[0], p[1], 0x5410u), prmt(p[2], p[3], 0x5410u), prmt(p[0], p[1], 0x7632u),
                              prmt(p[2], p[3], 0x7632u));
        }
        uint4 *dst = w_out + n * words_per_row + j;
        if (WIDE) {
            st_stream32(dst, o[0], o[1]);
        } else {  // output that is 16-byte aligned only
            dst[0] = o[0];
            dst[1] = o[1];
        }
    }
}

template <bool BF16, bool WIDE, int ROWS>
static cudaError_t dequant_dispatch(int zmode, dim3 grid, cudaStream_t s, const uint32_t *qw, const uint16_t *sc, const void *z,
                                    int zc, uint4 *out, int64_t N, int words_per_row, int group_words) {
    auto *fn = zmode == QF_ZERO_CONST ? dequant_kernel<BF16, QF_ZERO_CONST, WIDE, ROWS>
               : zmode == QF_ZERO_U4  ? dequant_kernel<BF16, QF_ZERO_U4, WIDE, ROWS>
                                      : dequant_kernel<BF16, QF_ZERO_I8, WIDE, ROWS>;
    return launch_kernel(fn, grid, dim3(256), 0, s, pdl_enabled(), qw, sc, z, zc, out, N, words_per_row, group_words);
}

int launch_dequant(qf_ctx *ctx, const qf_linear_desc *d, const void *qw, const void *scales, const void *zeros,
                   void *w_out, cudaStream_t s) {
    if (d->N == 0) return QF_OK;
    const int64_t words = d->K / 8;
    const int64_t cols = (words + 63) / 64;
    const int per = dequant_rows(d->zero_mode, d->N, d->K);
    const int64_t rows = (d->N + 8 * per - 1) / (8 * per), planes = (rows + 65534) / 65535;
    const dim3 grid((unsigned)cols, (unsigned)((rows + planes - 1) / planes), (unsigned)planes);
    const bool wide = (uintptr_t)w_out % 32 == 0;
    const bool bf16 = d->act_dtype == QF_BF16;
    auto *fn = per == 4 ? (bf16 ? (wide ? dequant_dispatch<true, true, 4> : dequant_dispatch<true, false, 4>)
                                : (wide ? dequant_dispatch<false, true, 4> : dequant_dispatch<false, false, 4>))
                        : (bf16 ? (wide ? dequant_dispatch<true, true, 2> : dequant_dispatch<true, false, 2>)
                                : (wide ? dequant_dispatch<false, true, 2> : dequant_dispatch<false, false, 2>));
    return launched(ctx, fn(d->zero_mode, grid, s, (const uint32_t *)qw, (const uint16_t *)scales, zeros, d->zero_const,
                            (uint4 *)w_out, d->N, (int)words, d->group_size / 8),
                    "dequant");
}

}  // namespace qf
