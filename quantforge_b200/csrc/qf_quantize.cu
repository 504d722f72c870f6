// Group-wise INT4 quantisation of a 16- or 32-bit weight [N, K]: codes, scales and zero points in one pass.
//
// The arithmetic is the statement of quantforge_b200/quantize.py in fp32, step for step as torch computes it on CUDA, so that
// codes, scales and zeros are the same bits as that gives on the same device:
//   asymmetric  scale = round16(max((wmax - wmin) * (1/15), 2^-14)), zero = clamp(rint(-wmin / scale), 0, 15)
//   symmetric   scale = round16(max(wabs * (1/7), 2^-14)),           zero = 8
//   code = clamp(rint(w / scale) + zero, 0, 15)
// On the CPU torch divides by 15 and 7; a scale there can be the next 16-bit number (about one in 10^4 f16 scales of fp32
// weights), and with it some codes.
// 2 bytes in and 1 byte out per 16-bit weight (the codes are one byte each, the packing is a separate call): 7.7 us for
// 4096 x 4096 at the copy rate. It takes 10.0 us; as elementwise passes over fp32 copies it took 300 us.
#include "qf_common.cuh"

namespace qf {

template <int DT>
__device__ __forceinline__ void load4(const void *w, int64_t i, float (&v)[4]) {  // i: a multiple of 4
    if constexpr (DT == QF_F32) {
        const float4 f = *(reinterpret_cast<const float4 *>(w) + (i >> 2));
        v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
    } else {
        const uint2 u = *(reinterpret_cast<const uint2 *>(w) + (i >> 2));
        const uint32_t h[4] = {u.x & 0xffffu, u.x >> 16, u.y & 0xffffu, u.y >> 16};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            v[k] = DT == QF_BF16 ? __uint_as_float(h[k] << 16) : __half2float(__ushort_as_half((unsigned short)h[k]));
    }
}

__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The two 16-bit values of a word, and minimum and maximum of both at once (exact: the results are inputs).
template <int DT>
__device__ __forceinline__ float low_half(uint32_t x) {
    return DT == QF_BF16 ? __uint_as_float(x << 16) : __half2float(__ushort_as_half((unsigned short)(x & 0xffffu)));
}
template <int DT>
__device__ __forceinline__ float high_half(uint32_t x) {
    return DT == QF_BF16 ? __uint_as_float(x & 0xffff0000u) : __half2float(__ushort_as_half((unsigned short)(x >> 16)));
}
template <int DT>
__device__ __forceinline__ uint32_t min2_nan(uint32_t a, uint32_t b) {
    uint32_t r;
    if (DT == QF_BF16) asm("min.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("min.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
template <int DT>
__device__ __forceinline__ uint32_t max2_nan(uint32_t a, uint32_t b) {
    uint32_t r;
    if (DT == QF_BF16) asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

struct GroupParams {
    float scale;  // after rounding to the stored type
    float rcp;    // 1 / scale, rounded
    float zero;
    uint16_t scale_bits;
    bool plain;   // quotients of the group's values need no division, see quotient
};

// w / scale as a division rounds it, by the reciprocal. The product q0 is within 2 ulp of the quotient; its residual w - scale * q0 is a
// multiple of ulp(q0) * ulp(scale) and less than 2 ulp(q0) * scale, a number of 13 bits as a stored scale has 11 at most, so one fused
// operation gives it exactly; q0 + residual * rcp is then off by 2^-23 ulp before its own rounding. No quotient by an 11-bit number is
// that near to a rounding boundary without being on it (the distance is at least 2^-11 of half an ulp, or 0), so the rounding is the
// division's. Ties of a group's values, w = (k + 1/2) scale, one in 500 for bf16 weights, come out as ties.
__device__ __forceinline__ float quotient(float w, float scale, float rcp) {
    const float q0 = w * rcp;
    return fmaf(fmaf(-scale, q0, w), rcp, q0);
}

template <bool SYM>
__device__ __forceinline__ GroupParams group_params(float lo, float hi, int scale_dtype) {
    GroupParams g;
    float s = SYM ? max_nan(hi, -lo) * (1.0f / 7.0f) : (hi - lo) * (1.0f / 15.0f);
    s = max_nan(s, 6.103515625e-05f);
    if (scale_dtype == QF_BF16) {
        const __nv_bfloat16 b = __float2bfloat16_rn(s);
        g.scale_bits = __bfloat16_as_ushort(b);
        g.scale = __bfloat162float(b);
    } else {
        const __half h = __float2half_rn(s);
        g.scale_bits = __half_as_ushort(h);
        g.scale = __half2float(h);
    }
    g.rcp = 1.0f / g.scale;
    // (false for infinities and NaN as well, and where the reciprocal could be subnormal; 256: codes are cut out of 16 bits)
    g.plain = fmaxf(fabsf(lo), fabsf(hi)) * g.rcp < 256.0f && g.scale < 1e30f;
    if (SYM) {
        g.zero = 8.0f;
    } else {
        const float z = rintf(g.plain ? quotient(-lo, g.scale, g.rcp) : -lo / g.scale);
        g.zero = fminf(fmaxf(z, 0.0f), 15.0f);
    }
    return g;
}

// code = clamp(rint(w / scale) + zero, 0, 15). Adding 1.5 * 2^23 rounds to the nearest even integer and leaves it in the low bits.
constexpr float kRound = 12582912.0f;
__device__ __forceinline__ uint32_t code_exact(float w, const GroupParams &g) {
    return (uint32_t)(int)fminf(fmaxf(rintf(w / g.scale) + g.zero, 0.0f), 15.0f);
}
// Two fp32 values in a 64-bit register: one instruction works on both.
__device__ __forceinline__ uint64_t f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void split_f32x2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Four codes, one per byte. Quotients and roundings are made for two values at a time in fp32, zero point and clamp for two in 16 bits.
// (With the product alone, and the division where that comes near to a half, a warp of bf16 weights took that way for one in four of
// its 128 values: a fifth of all instructions, and bound by them 4096 x 4096 took 13.6 us instead of 10.0.)
__device__ __forceinline__ uint32_t codes4(const float *v, const GroupParams &g) {
    if (!g.plain) return code_exact(v[0], g) | code_exact(v[1], g) << 8 | code_exact(v[2], g) << 16 | code_exact(v[3], g) << 24;
    const uint64_t rcp = f32x2(g.rcp, g.rcp), minus = f32x2(-g.scale, -g.scale), round = f32x2(kRound, kRound);
    uint32_t m[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint64_t w = f32x2(v[2 * h], v[2 * h + 1]);
        const uint64_t q0 = mul_f32x2(w, rcp);
        const uint64_t r = add_f32x2(fma_f32x2(fma_f32x2(minus, q0, w), rcp, q0), round);
        float a, b;
        split_f32x2(r, a, b);
        m[2 * h] = __float_as_uint(a);
        m[2 * h + 1] = __float_as_uint(b);
    }
    const uint32_t zero = dup16((uint32_t)(int)g.zero);
    const uint32_t a = __viaddmin_s16x2_relu(prmt(m[0], m[1], 0x5410u), zero, 0x000f000fu);
    const uint32_t b = __viaddmin_s16x2_relu(prmt(m[2], m[3], 0x5410u), zero, 0x000f000fu);
    return prmt(a, b, 0x6420u);
}
__device__ __forceinline__ void codes16(const float (&v)[16], const GroupParams &g, uint32_t (&c)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = codes4(v + 4 * k, g);
}

// Groups of 128 (256, 512): eight (16, 32) lanes hold a group in registers, sixteen values each, so a warp works on four neighbouring groups of
// a row (1 KB in for 16-bit weights) and the scale's divisions and roundings are paid once per 512 weights. A block covers
// 16 rows of four groups, so that scales [G, N] leave as whole sectors; all its loads are in flight before the first is used.
// (32 rows with half of the loads ahead: 1.7 waves for 4096 x 4096. Alone, on weights not in L2, bf16 asymmetric / f16 symmetric:
// 15.9 / 12.2 -> 13.7 / 10.1 us, 14336 x 4096 47.1 / 36.0 -> 40.8 / 31.3; with quotients as above 10.0 / 9.1 and 31.2 / 29.4; all bytes at the
// copy rate 7.7 and 27.) Five blocks of 48 registers per SM for 16-bit weights (four 10.2 / 9.7, six 10.6 / 10.1, 32 rows a block 10.5 / 9.6); fp32
// ones need the registers (four blocks 12.8 us, five 14.4 before). The steps from 32 rows to this (16 rows, loads ahead, two fp32 values per instruction, extremes in one word,
// zero point by reciprocal) were measured together only.
// With a group per warp, four values a lane, the kernel was bound by issue slots (25.2 us for 4096 x 4096 bf16). Groups of 256 and 512 took 36.8
// and 36.1 us as blocks of their own, 10.0 so.
constexpr int QUANT_PASSES = 2;  // rows a warp works on
template <int DT, bool SYM, bool TALL, int LANES>
__global__ void __launch_bounds__(256, DT == QF_F32 ? 4 : 5) quantize_warp_kernel(const void *w, int64_t N, int64_t K, uint32_t *codes,
                                                          uint16_t *scales, int scale_dtype, int8_t *zeros) {
    griddep_begin();
    constexpr int ROWS = 8 * QUANT_PASSES;
    constexpr int GROUPS = 32 / LANES;  // of a warp
    __shared__ uint16_t s_scale[GROUPS][ROWS];
    __shared__ int8_t s_zero[GROUPS][ROWS];
    constexpr int VEC = DT == QF_F32 ? 4 : 8;  // values of a 16-byte load
    constexpr int LOADS = 16 / VEC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane / LANES, t = lane % LANES;  // group of the warp's, lane of the group
    const int64_t G = K / (16 * LANES);
    const int64_t gi = (int64_t)blockIdx.x * GROUPS + q;
    const int64_t n0 = TALL ? ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * ROWS : (int64_t)blockIdx.y * ROWS;
    const bool have = gi < G;
    const int64_t first = (n0 + warp) * K + gi * (16 * LANES);  // of the row of pass 0; a pass is 8 rows
    uint4 u[QUANT_PASSES][LOADS];
#pragma unroll
    for (int pass = 0; pass < QUANT_PASSES; ++pass)
#pragma unroll
        for (int l = 0; l < LOADS; ++l) {
            u[pass][l] = make_uint4(0u, 0u, 0u, 0u);
            if (have && n0 + pass * 8 + warp < N)  // neighbouring lanes take neighbouring 16-byte pieces
                u[pass][l] = reinterpret_cast<const uint4 *>(w)[(first + pass * 8 * K) / VEC + l * LANES + t];
        }
#pragma unroll
    for (int pass = 0; pass < QUANT_PASSES; ++pass) {
        const int row = pass * 8 + warp;
        float v[16], lo, hi;
        uint32_t lo2 = 0, hi2 = 0;  // 16-bit types: running minimum and maximum of two values at a time
#pragma unroll
        for (int l = 0; l < LOADS; ++l) {
            const uint32_t x[4] = {u[pass][l].x, u[pass][l].y, u[pass][l].z, u[pass][l].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (DT == QF_F32) {
                    v[l * 4 + k] = __uint_as_float(x[k]);
                } else {
                    lo2 = l + k == 0 ? x[0] : min2_nan<DT>(lo2, x[k]);
                    hi2 = l + k == 0 ? x[0] : max2_nan<DT>(hi2, x[k]);
                    v[l * 8 + 2 * k] = low_half<DT>(x[k]);
                    v[l * 8 + 2 * k + 1] = high_half<DT>(x[k]);
                }
            }
        }
        if constexpr (DT == QF_F32) {
            lo = hi = v[0];
#pragma unroll
            for (int k = 1; k < 16; ++k) lo = min_nan(lo, v[k]), hi = max_nan(hi, v[k]);
#pragma unroll
            for (int o = LANES / 2; o; o >>= 1) {
                lo = min_nan(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max_nan(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
        } else {
            // (minimum, -maximum) in one word: the minimum of such words, over the halves and over the lanes, is both
            hi2 ^= 0x80008000u;
            uint32_t e = min2_nan<DT>(prmt(lo2, hi2, 0x5410u), prmt(lo2, hi2, 0x7632u));
#pragma unroll
            for (int o = LANES / 2; o; o >>= 1) e = min2_nan<DT>(e, __shfl_xor_sync(0xffffffffu, e, o));
            lo = low_half<DT>(e);
            hi = -high_half<DT>(e);
        }
        const GroupParams g = group_params<SYM>(lo, hi, scale_dtype);
        uint32_t c[4];
        codes16(v, g, c);
        if (have && n0 + row < N) {
            uint32_t *dst = codes + (first + pass * 8 * K) / 4;
#pragma unroll
            for (int l = 0; l < LOADS; ++l) {
                if constexpr (VEC == 8) reinterpret_cast<uint2 *>(dst)[l * LANES + t] = make_uint2(c[2 * l], c[2 * l + 1]);
                else dst[l * LANES + t] = c[l];
            }
        }
        if (t == 0) {
            s_scale[q][row] = g.scale_bits;
            s_zero[q][row] = (int8_t)(int)g.zero;
        }
    }
    __syncthreads();
    const int64_t n = n0 + lane;
    const int64_t go = (int64_t)blockIdx.x * GROUPS + warp;
    if (warp < GROUPS && lane < ROWS && go < G && n < N) {
        scales[go * N + n] = s_scale[warp][lane];
        if (!SYM) zeros[go * N + n] = s_zero[warp][lane];
    }
}

// Larger groups, multiples of 16 values: a block per (row, group), sixteen values a thread in registers as above; what a block of the
// largest kind cannot hold is read twice, the second time from L1 or L2. 4096 x 4096 bf16, four values a thread at a time in
// two passes -> this: groups of 1024 38.7 -> 14.1 us, 2048 27.0 -> 14.2, 4096 19.3 -> 15.2; 1024 x 28672 in one group a row 45.5 -> 21.6.
// Eight sizes of blocks, because threads without values cost nearly what the others do: with 64, 128, 256 and 512 alone rows of 4112 to 6400 and of 8208
// took as long as those of 8192, longer than in two passes (2048 x 5120 f16 17.7 us, so 10.1, in two passes 13.1; 1024 x 8208 fp32 15.9, 12.0 and 12.8).
template <int DT, bool SYM, int THREADS>
__global__ void __launch_bounds__(THREADS, DT == QF_F32 ? (1024 + THREADS / 2) / THREADS : THREADS == 448 ? 3 : 1280 / THREADS)
quantize_block_kernel(const void *w, int64_t N, int64_t K, int group, uint32_t *codes, uint16_t *scales, int scale_dtype, int8_t *zeros) {
    if (THREADS >= 256) griddep_launch_dependents();  // (see quantize_group_kernel)
    griddep_wait();
    constexpr int VEC = DT == QF_F32 ? 4 : 8;  // values of a 16-byte load
    constexpr int LOADS = 16 / VEC, TILE = THREADS * 16;
    __shared__ float s_lo[THREADS / 32], s_hi[THREADS / 32];
    const int64_t G = K / group;
    const int64_t n = blockIdx.x / G, gi = blockIdx.x % G;
    const int64_t base = n * K + gi * group;
    const uint4 *src = reinterpret_cast<const uint4 *>(w) + base / VEC;
    const int pieces = group / VEC;
    uint4 u[LOADS];
    auto load = [&](int first) {
#pragma unroll
        for (int l = 0; l < LOADS; ++l) {
            const int i = first / VEC + l * THREADS + (int)threadIdx.x;
            u[l] = i < pieces ? src[i] : src[0];  // (in place of what there is not, a value that is in the group anyway)
        }
    };
    float lo = __int_as_float(0x7f800000), hi = -lo;
    const int tiles = (group + TILE - 1) / TILE;
    // the last tile first: the first one stays in registers
    for (int tile = tiles - 1; tile >= 0; --tile) {
        load(tile * TILE);
        uint32_t lo2 = u[0].x, hi2 = u[0].x;
#pragma unroll
        for (int l = 0; l < LOADS; ++l) {
            const uint32_t x[4] = {u[l].x, u[l].y, u[l].z, u[l].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (DT == QF_F32) {
                    lo = min_nan(lo, __uint_as_float(x[k]));
                    hi = max_nan(hi, __uint_as_float(x[k]));
                } else {
                    lo2 = min2_nan<DT>(lo2, x[k]);
                    hi2 = max2_nan<DT>(hi2, x[k]);
                }
            }
        }
        if constexpr (DT != QF_F32) {
            lo = min_nan(lo, min_nan(low_half<DT>(lo2), high_half<DT>(lo2)));
            hi = max_nan(hi, max_nan(low_half<DT>(hi2), high_half<DT>(hi2)));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        lo = min_nan(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max_nan(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (THREADS > 32) {
        if ((threadIdx.x & 31) == 0) s_lo[threadIdx.x >> 5] = lo, s_hi[threadIdx.x >> 5] = hi;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < THREADS / 32; ++i) lo = min_nan(lo, s_lo[i]), hi = max_nan(hi, s_hi[i]);
    }
    const GroupParams g = group_params<SYM>(lo, hi, scale_dtype);
    uint32_t *dst = codes + base / 4;
#pragma unroll 1
    for (int tile = 0; tile < tiles; ++tile) {
        if (tile > 0) load(tile * TILE);
        float v[16];
#pragma unroll
        for (int l = 0; l < LOADS; ++l) {
            const uint32_t x[4] = {u[l].x, u[l].y, u[l].z, u[l].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (DT == QF_F32) {
                    v[l * 4 + k] = __uint_as_float(x[k]);
                } else {
                    v[l * 8 + 2 * k] = low_half<DT>(x[k]);
                    v[l * 8 + 2 * k + 1] = high_half<DT>(x[k]);
                }
            }
        }
        uint32_t c[4];
        codes16(v, g, c);
#pragma unroll
        for (int l = 0; l < LOADS; ++l) {
            const int i = tile * TILE / VEC + l * THREADS + (int)threadIdx.x;
            if (i >= pieces) continue;
            if constexpr (VEC == 8) reinterpret_cast<uint2 *>(dst)[i] = make_uint2(c[2 * l], c[2 * l + 1]);
            else dst[i] = c[l];
        }
    }
    if (threadIdx.x == 0) {
        scales[gi * N + n] = g.scale_bits;
        if (!SYM) zeros[gi * N + n] = (int8_t)(int)g.zero;
    }
}

// The other group sizes, multiples of 4: a block per (row, group), two passes over the group (the second one reads it from L1 or L2). Only
// blocks of 256 threads let the next kernel in early: the GPU takes one such signal a nanosecond, and there is one per block, so that in
// smaller blocks they were all the time (4096 x 4096 bf16 in groups of 64: 270.8 us instead of 137.6).
template <int DT, bool SYM>
__global__ void __launch_bounds__(256) quantize_group_kernel(const void *w, int64_t N, int64_t K, int group,
                                                             uint32_t *codes, uint16_t *scales,
                                                             int scale_dtype, int8_t *zeros) {
    if (blockDim.x == 256) griddep_launch_dependents();
    griddep_wait();
    __shared__ float s_lo[8], s_hi[8];
    const int64_t G = K / group;
    const int64_t n = blockIdx.x / G, gi = blockIdx.x % G;
    const int64_t base = n * K + gi * group;
    float lo = __int_as_float(0x7f800000), hi = -lo;
    for (int i = threadIdx.x * 4; i < group; i += blockDim.x * 4) {
        float v[4];
        load4<DT>(w, base + i, v);
#pragma unroll
        for (int k = 0; k < 4; ++k) lo = min_nan(lo, v[k]), hi = max_nan(hi, v[k]);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        lo = min_nan(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max_nan(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) s_lo[threadIdx.x >> 5] = lo, s_hi[threadIdx.x >> 5] = hi;
    __syncthreads();
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) lo = min_nan(lo, s_lo[i]), hi = max_nan(hi, s_hi[i]);
    const GroupParams g = group_params<SYM>(lo, hi, scale_dtype);
    for (int i = threadIdx.x * 4; i < group; i += blockDim.x * 4) {
        float v[4];
        load4<DT>(w, base + i, v);
        codes[(base + i) / 4] = codes4(v, g);
    }
    if (threadIdx.x == 0) {
        scales[gi * N + n] = g.scale_bits;
        if (!SYM) zeros[gi * N + n] = (int8_t)(int)g.zero;
    }
}

template <int DT, bool SYM>
static cudaError_t quantize_launch(const void *w, int64_t N, int64_t K, int group, uint32_t *codes, uint16_t *scales,
                                   int scale_dtype, int8_t *zeros, cudaStream_t s) {
    constexpr int ROWS = 8 * QUANT_PASSES;
    if (group == 128 || group == 256 || group == 512) {
        // Blocks of rows in y and, where there are more than 65535 of them, in z: 1.1 million rows of 128 297 us, a block per group
        // as below 572. (With z in the address everywhere, symmetric 4096 x 14336 took 39.3 us instead of 38.6.)
        const int64_t blocks = (N + ROWS - 1) / ROWS, z = (blocks + 65534) / 65535;
        const dim3 grid((unsigned)((K + 511) / 512), (unsigned)((blocks + z - 1) / z), (unsigned)z);
        auto *fn = group == 128   ? (z > 1 ? quantize_warp_kernel<DT, SYM, true, 8> : quantize_warp_kernel<DT, SYM, false, 8>)
                   : group == 256 ? (z > 1 ? quantize_warp_kernel<DT, SYM, true, 16> : quantize_warp_kernel<DT, SYM, false, 16>)
                                  : (z > 1 ? quantize_warp_kernel<DT, SYM, true, 32> : quantize_warp_kernel<DT, SYM, false, 32>);
        return launch_kernel(fn, grid, dim3(256), 0, s, pdl_enabled(), w, N, K, codes, scales, scale_dtype, zeros);
    }
    if (group > 512 && group % 16 == 0 && group <= 1 << 24) {
        // the fewest threads whose tiles hold the group (448 in up to two tiles: of four, 512 x 28672 f16 13.3 us instead of 12.4)
        const int tiles = (group + 8191) / 8192, need = (group + 16 * tiles - 1) / (16 * tiles);
        const int threads = need <= 64 ? 64 : need <= 128 ? 128 : need <= 192 ? 192 : need <= 256 ? 256 : need <= 320 ? 320 : need <= 384 ? 384 : need <= 448 && tiles <= 2 ? 448 : 512;
        auto *fn = threads == 64    ? quantize_block_kernel<DT, SYM, 64>
                   : threads == 128 ? quantize_block_kernel<DT, SYM, 128>
                   : threads == 192 ? quantize_block_kernel<DT, SYM, 192>
                   : threads == 256 ? quantize_block_kernel<DT, SYM, 256>
                   : threads == 320 ? quantize_block_kernel<DT, SYM, 320>
                   : threads == 384 ? quantize_block_kernel<DT, SYM, 384>
                   : threads == 448 ? quantize_block_kernel<DT, SYM, 448>
                                    : quantize_block_kernel<DT, SYM, 512>;
        return launch_kernel(fn, dim3((unsigned)(N * (K / group))), dim3(threads), 0, s, pdl_enabled(), w, N, K, group, codes, scales, scale_dtype, zeros);
    }
    const int threads = group >= 1024 ? 256 : group >= 512 ? 128 : group >= 256 ? 64 : 32;
    return launch_kernel(quantize_group_kernel<DT, SYM>, dim3((unsigned)(N * (K / group))), dim3(threads), 0, s, pdl_enabled(), w, N, K,
                         group, codes, scales, scale_dtype, zeros);
}

int launch_quantize(qf_ctx *ctx, const void *w, int dtype, int64_t N, int64_t K, int group, bool symmetric, void *codes,
                    void *scales, int scale_dtype, void *zeros, cudaStream_t s) {
    auto *fn = dtype == QF_F16    ? (symmetric ? quantize_launch<QF_F16, true> : quantize_launch<QF_F16, false>)
               : dtype == QF_BF16 ? (symmetric ? quantize_launch<QF_BF16, true> : quantize_launch<QF_BF16, false>)
                                  : (symmetric ? quantize_launch<QF_F32, true> : quantize_launch<QF_F32, false>);
    return launched(ctx, fn(w, N, K, group, (uint32_t *)codes, (uint16_t *)scales, scale_dtype, (int8_t *)zeros, s), "quantize");
}

}  // namespace qf
