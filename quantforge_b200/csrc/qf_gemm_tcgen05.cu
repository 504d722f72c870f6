// K3: W4A16 GEMM on the 5th-generation tensor cores (tcgen05), weights dequantised in the mainloop.
//
// Computes Y^T = W . X^T tile by tile so that the DEQUANTISED WEIGHTS are the MMA's A operand and
// live only in tensor memory (TMEM):
//   MMA M = 128 output features (weight rows, one per TMEM lane)
//   MMA N = the batch tile's rows of X, a multiple of 16 up to the instantiation's BN (16..256)
//   MMA K = 16  per instruction, BK codes per pipeline stage
//
// Roles inside a CTA (320 threads):
//   warps 0-3, 4-7 : two converter groups, alternating k-blocks. Thread t of a group owns weight row
//                    n0 + t: it reads the row's packed codes from the TMA-staged shared-memory tile,
//                    converts them with lop3 / packed 16-bit arithmetic (zero and scale of its own
//                    row and group held in registers), and writes the 16-bit operand straight into
//                    TMEM lane t with tcgen05.st.  The same threads run the epilogue
//                    (tcgen05.ld -> fp32 tile in shared memory -> whole output rows, or split-K partials).
//   warp 8         : TMA producer (one elected thread): packed-weight tile and X tile per stage.
//   warp 9         : TMEM allocation and, one elected thread, tcgen05.mma issue: A from TMEM,
//                    B (= X tile, K-major, 128-byte swizzle) from shared memory, fp32 accumulate in TMEM.
// Every mbarrier wait is bounded: on expiry the CTA raises an abort flag, records QF_ERR_TIMEOUT in
// the context's status word, drains its own TMA copies, frees its TMEM and returns.
// Every CTA loads its own tiles (plain TMA loads). Wide tiles run as CTA pairs, see gemm_kernel. Split-K of narrow tiles over
// 2..8 blocks runs as a thread-block cluster whose blocks sum their partial tiles through distributed shared memory; other
// splits use global partial tiles and an arrival counter. All cluster barriers are passed by every block, aborted or not.
#include <cuda.h>

#include <cstdlib>

#include "qf_common.cuh"
#include "qf_mbar.cuh"
#include "qf_tcgen05.cuh"

namespace qf {

// ---------------------------------------------------------------------------------------------
// configuration per batch-tile width
// ---------------------------------------------------------------------------------------------
// PAIR: two CTAs (weight tiles 2i and 2i + 1 of one batch tile) run their MMAs as one of 256 weight rows.
template <int BN, bool PAIR = false>
struct GemmCfg {
    static constexpr int BK = (BN <= 128 || PAIR) ? 128 : 64;   // codes per k-block
    static constexpr int X_ROWS = PAIR ? BN / 2 : BN;            // batch rows a CTA stages (at most)
    static constexpr int W_ROW_BYTES = BK / 2;                   // 64 or 32
    static constexpr int W_STAGE_BYTES = 128 * W_ROW_BYTES;      // 8 KB or 4 KB
    static constexpr int X_BOX_BYTES = X_ROWS * 128;             // one 64-element box
    static constexpr int X_STAGE_BYTES = X_BOX_BYTES * (BK / 64);
    static constexpr int STAGE_BYTES = W_STAGE_BYTES + X_STAGE_BYTES;
    static constexpr int STAGES = BN == 16 || (PAIR && BN == 128) ? 8 : BN == 32 ? 6 : BN == 64 ? 4 : 5;
    static constexpr int NA = BN <= 64 ? 3 : 4;                  // A operand buffers in TMEM
    static constexpr int A_COLS = BK / 2;                        // 32-bit TMEM columns per A buffer
    static constexpr int TMEM_COLS = (BN + NA * A_COLS) <= 256 ? 256 : 512;
    static constexpr int CTAS_PER_SM = BN <= 64 ? 2 : 1;
    static_assert(BN * 512 <= STAGES * STAGE_BYTES, "the epilogue stages the fp32 tile in the pipeline's memory");
    static constexpr int SZ_BYTES = 512;                          // per stage: 256 B scales + up to 128 B zeros
    static constexpr int SMEM_BYTES =
        STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/ + STAGES * SZ_BYTES;
};

constexpr int GEMM_THREADS = 320;

struct GemmParams {
    const uint16_t *scales;
    const void *zeros;
    void *Y;
    float *partial;
    int *counters;
    int *status;  // host-mapped status word
    int64_t M, N, K;
    int group_size;
    int zero_mode, zero_const;
    int out_dtype;
    int bn;                // batch rows of a tile: a multiple of 16, at most the instantiation's BN (the MMA's N)
    int kblocks;           // K / BK
    int kblocks_per_split;
    int split_k;
    int interleaved;       // weight nibble order inside a word: 0 canonical, 1 pair-interleaved
    int tiled;             // 1: weights stored tile-major (QF_LAYOUT_TILED)
    int cluster_reduce;    // 1: the split_k blocks of a tile form a thread-block cluster and sum their partial
                           //    tiles through distributed shared memory (no global partials, no counters)
    const void *residual;  // QF_EPI_RESIDUAL_ADD: R[M, N] in out_dtype
    int epilogue;          // qf_epilogue (plain instantiations only)
    int early;             // follows_linear: weights, scales and zeros may be read before the dependency wait
};

__device__ __forceinline__ float silu_mul(float gate, float up) { return gate / (1.f + expf(-gate)) * up; }
// CNT (4 or 8) consecutive elements of the output type, as vectors: element offsets are multiples of CNT, the base is 16-byte aligned
// and rows have a multiple of 16 elements, 32 bytes of a 16-bit type, so that vectors of up to 16 bytes are aligned.
template <int CNT>
__device__ __forceinline__ void store_vec(void *Y, int out_dtype, int64_t o, const float (&v)[CNT]) {
    if (out_dtype == QF_F32) {
        float4 *dst = reinterpret_cast<float4 *>(reinterpret_cast<float *>(Y) + o);
#pragma unroll
        for (int i = 0; i < CNT / 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        return;
    }
    uint32_t r[CNT / 2];
#pragma unroll
    for (int i = 0; i < CNT / 2; ++i) {
        if (out_dtype == QF_F16) {
            const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            r[i] = *reinterpret_cast<const uint32_t *>(&h);
        } else {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            r[i] = *reinterpret_cast<const uint32_t *>(&h);
        }
    }
    uint16_t *dst = reinterpret_cast<uint16_t *>(Y) + o;
    if constexpr (CNT == 8) *reinterpret_cast<uint4 *>(dst) = make_uint4(r[0], r[1], r[2], r[3]);
    else *reinterpret_cast<uint2 *>(dst) = make_uint2(r[0], r[1]);
}
template <int CNT>
__device__ __forceinline__ void add_residual(const void *R, int out_dtype, int64_t o, float (&v)[CNT]) {
    if (out_dtype == QF_F32) {
        const float4 *src = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(R) + o);
#pragma unroll
        for (int i = 0; i < CNT / 4; ++i) {
            const float4 a = src[i];
            v[4 * i] += a.x;
            v[4 * i + 1] += a.y;
            v[4 * i + 2] += a.z;
            v[4 * i + 3] += a.w;
        }
        return;
    }
    uint32_t r[CNT / 2];
    const uint16_t *src = reinterpret_cast<const uint16_t *>(R) + o;
    if constexpr (CNT == 8) {
        const uint4 a = *reinterpret_cast<const uint4 *>(src);
        r[0] = a.x, r[1] = a.y, r[2] = a.z, r[3] = a.w;
    } else {
        const uint2 a = *reinterpret_cast<const uint2 *>(src);
        r[0] = a.x, r[1] = a.y;
    }
#pragma unroll
    for (int i = 0; i < CNT / 2; ++i) {
        const float2 f = out_dtype == QF_F16 ? __half22float2(*reinterpret_cast<const __half2 *>(&r[i]))
                                             : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&r[i]));
        v[2 * i] += f.x;
        v[2 * i + 1] += f.y;
    }
}
// CNT finished outputs of batch row m, weight rows n.. (n a multiple of CNT), with the plain or residual epilogue.
template <int CNT>
__device__ __forceinline__ void gemm_store(const GemmParams &p, int64_t m, int64_t n, float (&v)[CNT]) {
    const int64_t o = m * p.N + n;
    if (p.epilogue == QF_EPI_RESIDUAL_ADD) add_residual<CNT>(p.residual, p.out_dtype, o, v);
    store_vec<CNT>(p.Y, p.out_dtype, o, v);
}
// QF_EPI_SILU_MUL: weight rows n.. (n % 16 < 8) are gate rows, n+8.. the matching up rows; output column
// (n / 16) * 8 + n % 8 of Y[M, N/2].
template <int CNT>
__device__ __forceinline__ void gemm_store_silu(const GemmParams &p, int64_t m, int64_t n, const float (&g)[CNT],
                                                const float (&u)[CNT]) {
    float v[CNT];
#pragma unroll
    for (int i = 0; i < CNT; ++i) v[i] = silu_mul(g[i], u[i]);
    store_vec<CNT>(p.Y, p.out_dtype, m * (p.N >> 1) + (n >> 4) * 8 + (n & 7), v);
}
__device__ __forceinline__ void gemm_store4(const GemmParams &p, int64_t m, int64_t n, float4 a) {
    float v[4] = {a.x, a.y, a.z, a.w};
    gemm_store<4>(p, m, n, v);
}
// Four residual elements as they lie in memory (16-bit types: in x and y), and added.
__device__ __forceinline__ uint4 load4_raw(const void *R, int out_dtype, int64_t o) {
    if (out_dtype == QF_F32) return *reinterpret_cast<const uint4 *>(reinterpret_cast<const float *>(R) + o);
    const uint2 v = *reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(R) + o);
    return make_uint4(v.x, v.y, 0u, 0u);
}
__device__ __forceinline__ void gemm_store4(const GemmParams &p, int64_t m, int64_t n, float4 a, uint4 add) {
    float v[4] = {a.x, a.y, a.z, a.w};
    if (p.epilogue == QF_EPI_RESIDUAL_ADD) {
        if (p.out_dtype == QF_F32) {
            v[0] += __uint_as_float(add.x), v[1] += __uint_as_float(add.y), v[2] += __uint_as_float(add.z), v[3] += __uint_as_float(add.w);
        } else {
            const uint32_t r[2] = {add.x, add.y};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float2 f = p.out_dtype == QF_F16 ? __half22float2(*reinterpret_cast<const __half2 *>(&r[i]))
                                                       : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&r[i]));
                v[2 * i] += f.x;
                v[2 * i + 1] += f.y;
            }
        }
    }
    store_vec<4>(p.Y, p.out_dtype, m * p.N + n, v);
}
__device__ __forceinline__ void gemm_store4_silu(const GemmParams &p, int64_t m, int64_t n, float4 g, float4 u) {
    const float gv[4] = {g.x, g.y, g.z, g.w}, uv[4] = {u.x, u.y, u.z, u.w};
    gemm_store_silu<4>(p, m, n, gv, uv);
}

template <int CNT>
__device__ __forceinline__ void lds_f4(uint32_t addr, float (&v)[4 * CNT]) {
#pragma unroll
    for (int i = 0; i < CNT; ++i)
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(v[4 * i]), "=f"(v[4 * i + 1]), "=f"(v[4 * i + 2]), "=f"(v[4 * i + 3])
                     : "r"(addr + 16u * i)
                     : "memory");
}
// (c0,c4)(c1,c5)(c2,c6)(c3,c7) -> (c0,c1)(c2,c3)(c4,c5)(c6,c7)
__device__ __forceinline__ void reorder8(uint32_t (&p)[4]) {
    const uint32_t lo0 = prmt(p[0], p[1], 0x5410u), lo1 = prmt(p[2], p[3], 0x5410u);
    const uint32_t hi0 = prmt(p[0], p[1], 0x7632u), hi1 = prmt(p[2], p[3], 0x7632u);
    p[0] = lo0;
    p[1] = lo1;
    p[2] = hi0;
    p[3] = hi1;
}
// 4 packed words (32 codes along K) -> 16 registers of 16-bit pairs in natural k order.
template <bool BF16, bool INTER>
__device__ __forceinline__ void convert32(const uint4 &v, const ShortConvert<BF16> &conv, uint32_t (&out)[16]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t p[4];
        conv(w[j], p);            // p[i] = (nibble i, nibble i+4)
        if (!INTER) reorder8(p);  // nibble order c0 c2 c4 c6 c1 c3 c5 c7: pairs are already (c0,c1)(c2,c3)..
#pragma unroll
        for (int i = 0; i < 4; ++i) out[4 * j + i] = p[i];
    }
}

// ---------------------------------------------------------------------------------------------
// kernel
// ---------------------------------------------------------------------------------------------
// EXCH: finished tiles are exchanged across GPUs (sum or gather) before Y is written; `ar` then is an ArParams.
// The plain instantiations take an empty struct instead, so their parameter block and code stay what they were.
// RAGGED: the last weight tile has fewer than 128 rows (an instantiation of its own: the same in all cost the others 1 to 2 %).
// PAIR: the grid runs in clusters of two blocks along x (weight tiles 2i, 2i + 1). A block stages half of the batch tile's
// rows and its own weights; its converters report to the first block, whose MMA warp issues cta_group::2 MMAs of 256
// weight rows for both and signals completion to both. With one CTA per MMA a k-block of 64 codes and 256 rows moves 72 KB
// through a block's shared memory (36 KB in, 32 KB to the tensor core, 4 KB of codes to the converters), 562 cycles at
// 128 bytes a cycle and more than the 512 the MMAs take; in a pair it is 40 KB. M = 2048, 8192 x 28672: 777 -> 738 us;
// M = 777, 4096 x 4096: 28.9 -> 27.5 us.
template <bool BF16, int BN, bool INTER, bool EXCH, bool PAIR, bool RAGGED = false>
__global__ void __launch_bounds__(GEMM_THREADS, GemmCfg<BN, PAIR>::CTAS_PER_SM)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
            const GemmParams p, const typename ExchArg<EXCH>::type ar) {
    using C = GemmCfg<BN, PAIR>;
    static_assert(!(PAIR && EXCH) && !(RAGGED && (PAIR || EXCH)), "the exchange serves the narrow tiles, whole ones");
    constexpr int BK = C::BK;
    constexpr int STAGES = C::STAGES;
    constexpr int NA = C::NA;
    constexpr bool CLUSTER_OK = BN <= 64 && !EXCH;  // the cluster reduction serves the narrow split-K tiles

    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ int s_is_last;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem_base + STAGES * C::STAGE_BYTES;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto afull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
    auto aempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + NA + a); };
    const uint32_t dfull_bar = bar_base + 8u * (2 * STAGES + 2 * NA);
    auto w_stage = [&](int s) { return smem_base + (uint32_t)s * C::STAGE_BYTES; };
    auto x_stage = [&](int s) { return smem_base + (uint32_t)s * C::STAGE_BYTES + C::W_STAGE_BYTES; };
    auto sz_stage = [&](int s) { return bar_base + 256u + (uint32_t)s * C::SZ_BYTES; };

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int m_tiles = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x;
    const int m_tile = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x;
    const int n_tile = PAIR ? (int)blockIdx.y * 2 + ((int)blockIdx.x & 1) : (int)blockIdx.y;
    const int split = blockIdx.z;
    const int kb0 = split * p.kblocks_per_split;
    const int kb1 = min(kb0 + p.kblocks_per_split, p.kblocks);
    const int nkb = kb1 - kb0;
    const int64_t n0 = (int64_t)n_tile * 128;
    const int64_t m0 = (int64_t)m_tile * p.bn;

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), PAIR ? 4 + 1 : 128 + 1);  // pair: one arrival per warp of a converter group
        }
        for (int a = 0; a < NA; ++a) {
            mbar_init(afull_bar(a), PAIR ? 2 * 4 : 128);      // of either block
            mbar_init(aempty_bar(a), 1);
        }
        mbar_init(dfull_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (RAGGED && n0 + 128 > p.N) {
        // scales and zeros of rows that there are not: no copy writes them
        for (int i = tid; i < STAGES * C::SZ_BYTES / 4; i += GEMM_THREADS)
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(bar_base + 256u + 4u * i), "r"(0u) : "memory");
        fence_proxy_async_shared();
    }
    if (warp == 8 && lane == 0) {
        tma_prefetch_desc(&tmap_w);
        tma_prefetch_desc(&tmap_x);
    }
    if (warp == 9) {
        tmem_alloc<PAIR>(smem_u32(&s_tmem_base), C::TMEM_COLS);
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();  // the other block's barriers exist
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    volatile int *abort_flag = &s_abort;
    if (p.early) griddep_launch_dependents();  // the next kernel may begin its own set-up and weight stream

    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    int producer_issued = 0;  // meaningful in the elected producer lane only
    if (warp == 8) {
        // ------------------------------ TMA producer ------------------------------
        // The whole warp runs the loop (uniform control flow); one elected lane issues the copies.
        const bool leader = elect_one();
        // (of a last tile of fewer than 128 rows what there is of scales and zeros; its codes' other rows are filled with zeros)
        const uint32_t sbytes = RAGGED ? (uint32_t)min((int64_t)128, p.N - n0) * 2u : 256u;
        const uint32_t zbytes = p.zero_mode == QF_ZERO_U4 ? sbytes / 4u : p.zero_mode == QF_ZERO_I8 ? sbytes / 2u : 0u;
        const int x_rows = PAIR ? p.bn >> 1 : p.bn;  // this block's share of the batch tile
        const int x_row0 = (int)m0 + (int)rank * x_rows;
        const uint32_t tx_bytes = C::W_STAGE_BYTES + (uint32_t)(BK / 64) * (uint32_t)x_rows * 128u + sbytes + zbytes;
        const int group_kb = p.group_size / BK;  // k-blocks per quantisation group (>= 1)
        const int gi = kb0 / group_kb;
        const uint8_t *sc_ptr = (const uint8_t *)(p.scales + n0) + (size_t)gi * p.N * 2;
        const size_t z_row = p.zero_mode == QF_ZERO_U4 ? (size_t)p.N / 2 : (size_t)p.N;
        const uint8_t *z_ptr =
            (const uint8_t *)p.zeros + (p.zero_mode == QF_ZERO_U4 ? (size_t)n0 / 2 : (size_t)n0) + (size_t)gi * z_row;
        const int w_row0 = p.tiled ? n_tile * (int)(p.K >> 7) * 128 : (int)n0;
        // issue_w is called for it = 0, 1, 2, ... in order: the sliver pointers advance incrementally
        int g_rem = kb0 % group_kb;
        // tile-major weights: rows of 64 bytes, the 128 rows of (n_tile, 128-code block) adjacent
        auto w_col = [&](int kb) { return !p.tiled ? kb * C::W_ROW_BYTES : (BK == 128) ? 0 : (kb & 1) * 32; };
        auto w_row = [&](int kb) { return !p.tiled ? w_row0 : w_row0 + ((kb * BK) >> 7) * 128; };
        auto issue_w = [&](int it, int s) {
            const int kb = kb0 + it;
            const uint32_t fb = full_bar(s);
            mbar_arrive_expect_tx(fb, tx_bytes);
            tma_load_2d(w_stage(s), &tmap_w, fb, w_col(kb), w_row(kb));
            bulk_load(sz_stage(s), sc_ptr, sbytes, fb);
            if (zbytes) bulk_load(sz_stage(s) + 256u, z_ptr, zbytes, fb);
            if (++g_rem == group_kb) {
                g_rem = 0;
                sc_ptr += (size_t)p.N * 2;
                z_ptr += z_row;
            }
        };
        auto issue_x = [&](int it, int s) {
            const int kb = kb0 + it;
#pragma unroll
            for (int b = 0; b < BK / 64; ++b)
                tma_load_2d(x_stage(s) + b * C::X_BOX_BYTES, &tmap_x, full_bar(s), kb * BK + b * 64, x_row0);
            producer_issued = it + 1;
        };
        // First pass over the ring. Behind a linear (follows_linear), weights, scales and zeros are requested before the
        // dependency wait and the activations after it; otherwise they go to L2 before the wait, and everything is requested
        // after it, stage by stage (weights of all stages first: 64 x 14336 x 4096 16.3 us instead of 15.9). A block that has
        // its SM to itself, or starts when others have left, finds the wait over or nearly so and prefetches nothing
        // (M = 2048, 8192 x 28672: 745 -> 737 us; M = 777, 4096 x 4096: 27.7 -> 27.1).
        const int npre = min(STAGES, nkb);
        const bool prefetch = C::CTAS_PER_SM > 1 &&
                              (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x < kSmCount * C::CTAS_PER_SM;
        if (leader) {
            for (int it = 0; it < npre; ++it) {
                if (p.early) {
                    issue_w(it, it);
                } else if (prefetch) {
                    const int dg = (kb0 + it) / group_kb - gi;  // groups behind the first one
                    tma_prefetch_2d(&tmap_w, w_col(kb0 + it), w_row(kb0 + it));
                    l2_prefetch(sc_ptr + (size_t)dg * p.N * 2, sbytes);
                    if (zbytes) l2_prefetch(z_ptr + (size_t)dg * z_row, zbytes);
                }
            }
        }
        griddep_wait();
        if (!p.early) griddep_launch_dependents();
        if (leader) {
            for (int it = 0; it < npre; ++it) {
                if (!p.early) issue_w(it, it);
                issue_x(it, it);
            }
        }
        int s = npre % STAGES;
        uint32_t ph = npre == STAGES ? 1u : 0u;
        for (int it = npre; it < nkb; ++it) {
            const bool ok = mbar_wait(empty_bar(s), ph ^ 1, abort_flag);
            if (!__all_sync(0xffffffffu, ok)) break;
            if (leader) {
                issue_w(it, s);
                issue_x(it, s);
            }
            if (++s == STAGES) {
                s = 0;
                ph ^= 1;
            }
        }
    } else if (warp == 9) {
        // ------------------------------ MMA issuer ------------------------------
        // One thread (of a pair: of the first block) runs the loop. It waits once per k-block: the converters reported after
        // they had seen the stage's copies (weights and X share a barrier) arrive.
        // (As a whole warp with two waits and a vote on each, a k-block took about 100 cycles more of this warp and of the issue
        // slots that the converters need: a 6-layer step at 9 rows 594 -> 582 us, 32 layers at 16 rows 1604 -> 1596 us.)
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) |
                                   ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)((PAIR ? 256 : 128) >> 4) << 24);
            const uint64_t desc0 = make_b_desc(x_stage(0));
            int s = 0, a = 0, it = 0;
            uint32_t aph = 0;
            for (; it < nkb; ++it) {
                if (!mbar_wait(afull_bar(a), aph, abort_flag)) break;
                tc_fence_after();
                const uint32_t a_tmem = tmem_base + BN + a * C::A_COLS;
                const uint64_t desc = desc0 + (uint32_t)s * (uint32_t)(C::STAGE_BYTES >> 4);
                umma_ts<PAIR>(tmem_base, a_tmem, desc, idesc, it > 0 ? 1u : 0u);
#pragma unroll
                for (int kk = 1; kk < BK / 16; ++kk)
                    umma_ts<PAIR>(tmem_base, a_tmem + kk * 8,
                                  desc + (uint32_t)(((kk >> 2) * C::X_BOX_BYTES + (kk & 3) * 32) >> 4), idesc, 1u);
                umma_commit<PAIR>(empty_bar(s));
                umma_commit<PAIR>(aempty_bar(a));
                if (++s == STAGES) s = 0;
                if (++a == NA) {
                    a = 0;
                    aph ^= 1;
                }
            }
            if (it == nkb) umma_commit<PAIR>(dfull_bar);
        }
        __syncwarp();
    } else {
        // ------------------------------ converters ------------------------------
        const int wg = warp >> 2;              // 0 or 1
        const int row = tid & 127;             // TMEM lane and weight row inside the tile
        const int64_t n = n0 + row;
        const uint32_t lane_taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        // swizzled 16-byte chunk positions of this row inside a weight stage
        const uint32_t row_off = (uint32_t)row * C::W_ROW_BYTES;
        const uint32_t sw = (BK == 128) ? ((row >> 1) & 3) : ((row >> 2) & 1);

        for (int it = wg; it < nkb; it += 2) {
            const int s = it % STAGES;
            const uint32_t ph = (it / STAGES) & 1;
            const int a = it % NA;
            const uint32_t aph = (it / NA) & 1;
            // warp-uniform outcome: the tcgen05.st below is warp-collective
            bool ready = mbar_wait(full_bar(s), ph, abort_flag);
            ready = ready && mbar_wait(aempty_bar(a), aph ^ 1, abort_flag);
            if (!__all_sync(0xffffffffu, ready)) break;
            tc_fence_after();
            // zero and scale of (this row, this k-block's group) from the stage's slivers
            ShortConvert<BF16> conv;
            {
                const uint32_t szb = sz_stage(s);
                uint32_t sbits;
                asm volatile("ld.shared.u16 %0, [%1];" : "=r"(sbits) : "r"(szb + 2u * row));
                int z = p.zero_const;
                if (p.zero_mode == QF_ZERO_U4) {
                    uint32_t zw;
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(zw) : "r"(szb + 256u + 4u * (row >> 3)));
                    z = (int)((zw >> (4 * (row & 7))) & 0xFu);
                } else if (p.zero_mode == QF_ZERO_I8) {
                    asm volatile("ld.shared.s8 %0, [%1];" : "=r"(z) : "r"(szb + 256u + row));
                }
                conv.set(z, sbits);
            }
            const uint32_t wbase = w_stage(s) + row_off;
            const uint32_t a_col = BN + a * C::A_COLS;
#pragma unroll
            for (int c = 0; c < C::W_ROW_BYTES / 16; ++c) {
                const uint4 v = lds128(wbase + (((uint32_t)c ^ sw) << 4));
                uint32_t out[16];
                convert32<BF16, INTER>(v, conv, out);
                tmem_st16(lane_taddr + a_col + c * 16, out);
            }
            if (BF16 && conv.wide) {
                // once more in the other form. Behind the ordinary path and rolled up: as a branch in front of it, or unrolled,
                // it cost that path its schedule or its registers (32 bf16 layers at 16 rows: 1688 and 1819 us)
                tmem_wait_st();
#pragma unroll 1
                for (int j = 0; j < C::W_ROW_BYTES / 4; ++j) {
                    uint32_t q[4];
                    dequant8<BF16>(lds32(wbase + ((((uint32_t)j >> 2) ^ sw) << 4) + ((uint32_t)j & 3u) * 4u), conv.zs, q);
                    if (!INTER) reorder8(q);
                    tmem_st4(lane_taddr + a_col + j * 4, q);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            fence_proxy_async_shared();  // this thread's reads of the stage, before the copy engine refills it
            if constexpr (PAIR) {
                __syncwarp();
                if (lane == 0) {
                    // at the first block's barrier; it also says that this block's half of X has arrived
                    mbar_arrive_cluster(dsmem_addr(afull_bar(a), 0u));
                    mbar_arrive(empty_bar(s));
                }
            } else {
                mbar_arrive(afull_bar(a));
                mbar_arrive(empty_bar(s));
            }
        }

        // ------------------------------ epilogue ------------------------------
        const bool ok = __all_sync(0xffffffffu, mbar_wait(dfull_bar, 0, abort_flag));
        tc_fence_after();
        if (ok) {
            // the activations this tile consumed were requested after the dependency wait, so the previous call on
            // this rank has finished and advanced the epoch
            unsigned ar_epoch = 0u;
            if constexpr (EXCH) ar_epoch = exch_read_epoch(ar);
            // TMEM -> fp32 tile [batch row][weight row] in the (now idle) pipeline stages, from where whole output rows
            // leave as 16-byte stores. Written straight from TMEM, one element per thread and store with the epilogue chosen per
            // element, a 128 x 256 tile took 23 700 cycles, a third of the whole K = 4096 tile (M = 2048, 8192 x 28672: 897 ->
            // 777 us; M = 777, 4096 x 4096: 35.6 -> 28.9 us; 64 x 14336 x 4096: 17.3 -> 15.9 us).
            // Split-K partial tiles that meet in global memory and exchanged tiles go there directly.
            const int cols_per_wg = p.bn >> 1;
            const int64_t Mp = (int64_t)m_tiles * p.bn;
            const bool to_partial = p.split_k > 1 && !(CLUSTER_OK && p.cluster_reduce);
            float *part = p.partial + ((int64_t)split * Mp + m0) * p.N + n;
#pragma unroll 1
            for (int c8 = 0; c8 < cols_per_wg >> 3; ++c8) {
                const int col = wg * cols_per_wg + c8 * 8;
                uint32_t r[8];
                if constexpr (RAGGED) __syncwarp();  // the last tile's stores may be half a warp's
                tmem_ld8(lane_taddr + col, r);
                tmem_wait_ld();
                if (to_partial) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (!RAGGED || n < p.N) __stcg(part + (int64_t)(col + j) * p.N, __uint_as_float(r[j]));
                } else if constexpr (EXCH) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int64_t m = m0 + col + j;
                        if (m < p.M) exch_push(ar, ar_epoch, (size_t)(m * p.N + n), __uint_as_float(r[j]));
                    }
                } else {
                    const uint32_t dst = smem_base + (uint32_t)(col * 128 + row) * 4u;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + j * 512u), "r"(r[j]) : "memory");
                }
            }
        }
    }

    // ------------------------------ teardown ------------------------------
    tc_fence_before();
    __syncthreads();
    if (CLUSTER_OK && p.cluster_reduce) {
        // Split-K inside a cluster: the split_k blocks of this tile are the blocks of one cluster (rank = split).
        // Every block, aborted or not, passes both cluster barriers, so no block can wait for one that left.
        if (s_abort && warp == 8 && producer_issued > 0) {
            int dummy = 0;
            volatile int *no_abort = &dummy;
            for (int it = max(0, producer_issued - STAGES); it < producer_issued; ++it)
                mbar_wait(full_bar(it % STAGES), (it / STAGES) & 1, no_abort);
        }
        if (s_abort && tid == 0) atomicExch(p.status, QF_ERR_TIMEOUT);
        cluster_sync_all();  // all partial tiles are in shared memory
        const int per = (32 * p.bn + p.split_k - 1) / p.split_k;  // float4 units of the tile that a block sums
        // Each block sums its share of the tile from all blocks in split order, a float4 unit per thread and round. Having read its last
        // units it says so, and writes them while the others are still at it. (One behind the other: 16 x 4096 x 1024 5.67 us instead of
        // 5.30, 16 x 4096 x 6144 8.45 instead of 8.03, 32 x 14336 x 4096 13.5 instead of 12.8, 64 x 4096 x 1024 6.79 instead of 6.34.)
        const bool silu = p.epilogue == QF_EPI_SILU_MUL;
        const int u_end = s_abort ? 0 : min(32 * p.bn, (split + 1) * per);
        auto mine = [&](int u) { return u < u_end && m0 + (u >> 5) < p.M && !(silu && (u & 2)) && (!RAGGED || n0 + (u & 31) * 4 < p.N); };
        auto total = [&](uint32_t at) {
            float4 v[8], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int sp = 0; sp < 8; ++sp)
                v[sp] = sp < p.split_k ? ld_dsmem_f4(dsmem_addr(at, (uint32_t)sp)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int sp = 0; sp < 8; ++sp) {
                sum.x += v[sp].x;
                sum.y += v[sp].y;
                sum.z += v[sp].z;
                sum.w += v[sp].w;
            }
            return sum;
        };
        int u = split * per + tid;
        if constexpr (BN > 16) {
#pragma unroll 1
            for (int left = per; left > GEMM_THREADS; left -= GEMM_THREADS, u += GEMM_THREADS)
                if (mine(u)) {
                    const uint32_t a = smem_base + (uint32_t)u * 16u;
                    const int64_t m = m0 + (u >> 5), n = n0 + (u & 31) * 4;
                    const float4 acc = total(a);
                    if (silu) gemm_store4_silu(p, m, n, acc, total(a + 32u));  // the matching up rows sit 8 rows further on
                    else gemm_store4(p, m, n, acc);
                }
        }
        const bool last = mine(u);
        const int64_t m = m0 + (u >> 5), n = n0 + (u & 31) * 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), up = acc;
        uint4 add = make_uint4(0u, 0u, 0u, 0u);
        if (last) {
            const uint32_t a = smem_base + (uint32_t)u * 16u;
            if (BN == 64 && p.epilogue == QF_EPI_RESIDUAL_ADD) add = load4_raw(p.residual, p.out_dtype, m * p.N + n);
            acc = total(a);
            if (silu) up = total(a + 32u);
        }
        cluster_arrive();
        if (last) {
            if (silu) gemm_store4_silu(p, m, n, acc, up);
            else if (BN == 64) gemm_store4(p, m, n, acc, add);
            else gemm_store4(p, m, n, acc);
        }
        cluster_wait();  // nobody leaves while its tile may still be read
    } else if (s_abort) {
        if (warp == 8 && producer_issued > 0) {
            // drain this CTA's own TMA copies before the shared memory goes away
            int dummy = 0;
            volatile int *no_abort = &dummy;
            for (int it = max(0, producer_issued - STAGES); it < producer_issued; ++it)
                mbar_wait(full_bar(it % STAGES), (it / STAGES) & 1, no_abort);
        }
        if (tid == 0) atomicExch(p.status, QF_ERR_TIMEOUT);
        __syncthreads();
    } else {
        if (!EXCH && p.split_k == 1) {
            const int rows = (int)min((int64_t)p.bn, p.M - m0);
            if (p.epilogue == QF_EPI_SILU_MUL) {
                for (int u = tid; u < rows * 8; u += GEMM_THREADS) {
                    const uint32_t a = smem_base + (uint32_t)u * 64u;  // 8 gate rows, then their 8 up rows
                    float v[16];
                    lds_f4<4>(a, v);
                    const float g[8] = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
                    const float up[8] = {v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15]};
                    gemm_store_silu<8>(p, m0 + (u >> 3), n0 + (u & 7) * 16, g, up);
                }
            } else {
                for (int u = tid; u < rows * 16; u += GEMM_THREADS) {
                    float v[8];
                    lds_f4<2>(smem_base + (uint32_t)u * 32u, v);
                    if (!RAGGED || n0 + (u & 15) * 8 < p.N) gemm_store<8>(p, m0 + (u >> 4), n0 + (u & 15) * 8, v);
                }
            }
        }
        bool final_cta = true;  // this CTA holds (or has pushed) the finished tile
        unsigned ar_epoch = 0u;
        if constexpr (EXCH) ar_epoch = exch_read_epoch(ar);
        if (p.split_k > 1) {
            // split-K: last CTA of this (m_tile, n_tile) sums the partial tiles in split order
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                int *cnt = p.counters + (int64_t)n_tile * m_tiles + m_tile;
                const int prev = atomicAdd(cnt, 1);
                s_is_last = (prev == p.split_k - 1);
                if (s_is_last) *cnt = 0;
            }
            __syncthreads();
            final_cta = s_is_last != 0;
            if (final_cta) {
                __threadfence();
                // Each thread owns 4 consecutive output columns (one 16-byte load per split) and keeps 4 splits in
                // flight, so the reduction is not a chain of dependent L2 round trips.
                const int64_t Mp = (int64_t)m_tiles * p.bn;
                const size_t split_stride = (size_t)Mp * p.N;
                for (int u = tid; u < 32 * p.bn; u += GEMM_THREADS) {
                    const int nl = (u & 31) * 4;
                    const int64_t m = m0 + (u >> 5);
                    const bool silu = !EXCH && p.epilogue == QF_EPI_SILU_MUL;
                    if (m < p.M && !(silu && (nl & 8)) && (!RAGGED || n0 + nl < p.N)) {
                        // sum over the splits of 4 consecutive output columns starting `off` columns into the row
                        auto sum4 = [&](int off) {
                            const float *base = p.partial + (size_t)m * p.N + n0 + nl + off;
                            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                            for (int sp0 = 0; sp0 < p.split_k; sp0 += 4) {
                                float4 v[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    v[j] = (sp0 + j < p.split_k)
                                               ? __ldcg(reinterpret_cast<const float4 *>(base + (size_t)(sp0 + j) * split_stride))
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    acc.x += v[j].x;
                                    acc.y += v[j].y;
                                    acc.z += v[j].z;
                                    acc.w += v[j].w;
                                }
                            }
                            return acc;
                        };
                        const float4 acc = sum4(0);
                        const int64_t o = m * p.N + n0 + nl;
                        if constexpr (EXCH) {
                            exch_push2(ar, ar_epoch, (size_t)o, acc.x, acc.y);
                            exch_push2(ar, ar_epoch, (size_t)o + 2, acc.z, acc.w);
                        } else if (silu) {
                            gemm_store4_silu(p, m, n0 + nl, acc, sum4(8));
                        } else {
                            gemm_store4(p, m, n0 + nl, acc);
                        }
                    }
                }
            }
        }
        if constexpr (EXCH) if (final_cta) {
            // Cross-GPU step: every element of the tile has been pushed to all ranks (above, or in the epilogue);
            // collect the other ranks' values for the same elements and write the output. The pairs carry their
            // own arrival token, so no block-level synchronisation separates the pushes from the collects.
            if (!exch_collect_tile(ar, ar_epoch, m0, p.bn, n0, 128, p.M, p.N, p.Y, p.out_dtype, tid, GEMM_THREADS,
                                   abort_flag))
                s_abort = 1;
            __syncthreads();
            if (tid == 0) exch_block_done(ar, ar_epoch, gridDim.x * gridDim.y, s_abort != 0);
        }
    }
    // a pair leaves together: MMAs read and signal both blocks, and both give back their TMEM
    if constexpr (PAIR) cluster_sync_all();
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc<PAIR>(tmem_base, C::TMEM_COLS);
    }
}


// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// Instantiation (widest batch tile) that serves a batch tile of bn rows.
static int gemm_tile_of(int bn) { return bn <= 16 ? 16 : bn <= 32 ? 32 : bn <= 64 ? 64 : bn <= 128 ? 128 : 256; }

constexpr bool gemm_has_pair(int bn) { return bn >= 128; }
constexpr bool gemm_has_exchange(int bn) { return bn <= 64; }  // the cross-GPU exchange serves decode batches only

template <bool BF16, int BN>
static cudaError_t gemm_set_attr() {
    const int bytes = GemmCfg<BN>::SMEM_BYTES;
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, false, false, false>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, true, false, false>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, false, false, false, true>, attr, bytes);
    if constexpr (gemm_has_exchange(BN)) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, false, true, false>, attr, bytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, true, true, false>, attr, bytes);
    }
    if constexpr (gemm_has_pair(BN)) {
        const int pair_bytes = GemmCfg<BN, true>::SMEM_BYTES;
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, false, false, true>, attr, pair_bytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_kernel<BF16, BN, true, false, true>, attr, pair_bytes);
    }
    return e;
}

int gemm_init(qf_ctx *ctx) {
    QF_CUDA_TRY(ctx, (gemm_set_attr<false, 16>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<false, 32>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<false, 64>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<false, 128>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<false, 256>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<true, 16>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<true, 32>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<true, 64>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<true, 128>()));
    QF_CUDA_TRY(ctx, (gemm_set_attr<true, 256>()));
    if (!ctx->host_status) {
        QF_CUDA_TRY(ctx, cudaHostAlloc((void **)&ctx->host_status, sizeof(int), cudaHostAllocMapped));
        *ctx->host_status = 0;
        QF_CUDA_TRY(ctx, cudaHostGetDevicePointer((void **)&ctx->dev_status, ctx->host_status, 0));
    }
    return QF_OK;
}

template <bool BF16, int BN, bool PAIR>
static int gemm_launch_bn(qf_ctx *ctx, const qf_linear_desc *d, const Plan &plan, const void *X, const void *qw,
                          GemmParams &p, cudaStream_t s, const ArParams *ar) {
    using C = GemmCfg<BN, PAIR>;
    CUtensorMap tw, tx;
    const bool tiled = d->weight_layout == QF_LAYOUT_TILED;
    int st = get_tensor_map(ctx, &tw, qw, 0, tiled ? 64 : (uint64_t)d->K / 2,
                            tiled ? (uint64_t)d->N * (uint64_t)(d->K / 128) : (uint64_t)d->N, C::W_ROW_BYTES, 128,
                            C::BK == 128 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    if (st != QF_OK) return st;
    st = get_tensor_map(ctx, &tx, X, 1, (uint64_t)d->K, (uint64_t)d->M, 64,
                        (uint32_t)(PAIR ? plan.bn / 2 : plan.bn), CU_TENSOR_MAP_SWIZZLE_128B);
    if (st != QF_OK) return st;
    p.bn = plan.bn;
    p.kblocks = (int)(d->K / C::BK);
    p.kblocks_per_split = plan.chunks_per_split;
    // a pair's blocks differ in x: the dimension along which cta_group::2 pairs them
    dim3 grid((unsigned)plan.m_tiles * (PAIR ? 2u : 1u), (unsigned)((d->N + 127) / 128) / (PAIR ? 2u : 1u), (unsigned)plan.split_k);
    const dim3 blk(GEMM_THREADS);
    cudaError_t le;
    if (ar) {
        if constexpr (gemm_has_exchange(BN) && !PAIR) {
            le = p.interleaved ? launch_kernel(gemm_kernel<BF16, BN, true, true, false>, grid, blk, C::SMEM_BYTES, s,
                                               pdl_enabled(), tw, tx, p, *ar)
                               : launch_kernel(gemm_kernel<BF16, BN, false, true, false>, grid, blk, C::SMEM_BYTES, s,
                                               pdl_enabled(), tw, tx, p, *ar);
        } else {
            return fail(ctx, QF_ERR_UNSUPPORTED, "the in-kernel exchange serves M <= 64");
        }
    } else {
        // 2..8 splits of a narrow tile: one thread-block cluster per tile sums the partial tiles on chip
        // Clusters are placed inside one GPC, which leaves block slots unused where the GPC's slot count is not a
        // multiple of the cluster size; a launch that no longer fits in one wave loses more than the on-chip
        // reduction gains (measured: 32 x 8, 80 x 3, 112 x 2 blocks fit; 48 x 6 = 288 of the 296 slots do not).
        unsigned cluster_z = 1;
        if (BN <= 64 && !PAIR && plan.split_k >= 2 && plan.split_k <= 8 && cluster_reduce_enabled()) {
            if ((int64_t)grid.x * grid.y * grid.z <= kClusterMaxBlocks) {
                p.cluster_reduce = 1;
                cluster_z = (unsigned)plan.split_k;
            }
        }
        const dim3 cluster(PAIR ? 2 : 1, 1, cluster_z);
        auto *fn = p.interleaved ? gemm_kernel<BF16, BN, true, false, PAIR> : gemm_kernel<BF16, BN, false, false, PAIR>;
        if constexpr (!PAIR)
            if (d->N % 128 != 0) fn = gemm_kernel<BF16, BN, false, false, false, true>;
        le = launch_kernel_cluster(fn, grid, blk, C::SMEM_BYTES, s, pdl_enabled(), cluster, tw, tx, p, NoExchange{});
    }
    note_linear(s);
    return launched(ctx, le, "GEMM");
}

template <bool BF16>
static int gemm_launch_dt(qf_ctx *ctx, const qf_linear_desc *d, const Plan &plan, const void *X, const void *qw,
                          GemmParams &p, cudaStream_t s, const ArParams *ar) {
    switch (gemm_tile_of(plan.bn)) {
        case 16: return gemm_launch_bn<BF16, 16, false>(ctx, d, plan, X, qw, p, s, ar);
        case 32: return gemm_launch_bn<BF16, 32, false>(ctx, d, plan, X, qw, p, s, ar);
        case 64: return gemm_launch_bn<BF16, 64, false>(ctx, d, plan, X, qw, p, s, ar);
        case 128:
            return plan.pair ? gemm_launch_bn<BF16, 128, true>(ctx, d, plan, X, qw, p, s, ar)
                             : gemm_launch_bn<BF16, 128, false>(ctx, d, plan, X, qw, p, s, ar);
        case 256:
            return plan.pair ? gemm_launch_bn<BF16, 256, true>(ctx, d, plan, X, qw, p, s, ar)
                             : gemm_launch_bn<BF16, 256, false>(ctx, d, plan, X, qw, p, s, ar);
        default: return fail(ctx, QF_ERR_BAD_ARG, "bad batch tile");
    }
}

int gemm_block_k(int bn, bool pair) { return bn <= 128 || pair ? 128 : 64; }

static int launch_gemm_impl(qf_ctx *ctx, const qf_linear_desc *d, const Plan &plan, const void *X, const void *qw,
                            const void *scales, const void *zeros, void *Y, const void *residual, void *ws,
                            cudaStream_t s, const ArParams *ar) {
    GemmParams p;
    p.residual = residual;
    p.epilogue = ar ? QF_EPI_NONE : d->epilogue;
    p.scales = (const uint16_t *)scales;
    p.zeros = zeros;
    p.Y = Y;
    p.counters = (int *)ws;
    p.partial = (float *)((char *)ws + plan.ws_counter_bytes);
    p.status = ctx->dev_status;
    p.M = d->M;
    p.N = d->N;
    p.K = d->K;
    p.group_size = d->group_size;
    p.zero_mode = d->zero_mode;
    p.zero_const = d->zero_const;
    p.out_dtype = d->out_dtype;
    p.split_k = plan.split_k;
    p.interleaved = d->weight_layout != QF_LAYOUT_CANONICAL;
    p.tiled = d->weight_layout == QF_LAYOUT_TILED;
    p.cluster_reduce = 0;
    p.early = follows_linear(s) ? 1 : 0;
    if (d->act_dtype == QF_BF16) return gemm_launch_dt<true>(ctx, d, plan, X, qw, p, s, ar);
    return gemm_launch_dt<false>(ctx, d, plan, X, qw, p, s, ar);
}

int launch_gemm(qf_ctx *ctx, const qf_linear_desc *d, const Plan &plan, const void *X, const void *qw,
                const void *scales, const void *zeros, void *Y, const void *residual, void *ws, cudaStream_t s) {
    return launch_gemm_impl(ctx, d, plan, X, qw, scales, zeros, Y, residual, ws, s, nullptr);
}

int launch_gemm_ar(qf_ctx *ctx, const qf_linear_desc *d, const Plan &plan, const void *X, const void *qw,
                   const void *scales, const void *zeros, void *Y, void *ws, cudaStream_t s, const ArParams &ar) {
    return launch_gemm_impl(ctx, d, plan, X, qw, scales, zeros, Y, nullptr, ws, s, &ar);
}

}  // namespace qf
