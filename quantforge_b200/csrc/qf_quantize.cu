// Group-wise INT4 quantisation of a 16- or 32-bit weight [N, K]: codes, scales and zero points in one pass.
//
// The arithmetic is the statement of quantforge_b200/quantize.py in fp32, step for step, so that codes, scales and zeros
// are the same bits whichever of the two computes them:
//   asymmetric  scale = round16(max((wmax - wmin) * (1/15), 2^-14)), zero = clamp(rint(-wmin / scale), 0, 15)
//   symmetric   scale = round16(max(wabs * (1/7), 2^-14)),           zero = 8
//   code = clamp(rint(w / scale) + zero, 0, 15)
// Bound by HBM: 2 bytes in and 1 byte out per weight (the codes are one byte each, the packing is a separate call). As
// elementwise passes over fp32 copies it took 300 us at 4096 x 4096.
#include "qf_common.cuh"

namespace qf {

template <int DT>
__device__ __forceinline__ void load4(const void *w, int64_t i, float (&v)[4]) {  // i: a multiple of 4
    if constexpr (DT == QF_F32) {
        const float4 f = __ldg(reinterpret_cast<const float4 *>(w) + (i >> 2));
        v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
    } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2 *>(w) + (i >> 2));
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

struct GroupParams {
    float scale;  // after rounding to the stored type
    float rcp;    // about 1 / scale
    float zero;
    uint16_t scale_bits;
};

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
    g.zero = SYM ? 8.0f : fminf(fmaxf(rintf(-lo / g.scale), 0.0f), 15.0f);
    return g;
}

// rint(w / scale). The product with the reciprocal is within 2 ulp of the quotient, so away from the rounding boundary
// (and for the quotients of at most a few tens that a group's own scale gives) it rounds to the same integer; near the
// boundary the division decides. Adding and subtracting 1.5 * 2^23 rounds to the nearest even integer.
__device__ __forceinline__ float round_quotient(float w, const GroupParams &g) {
    const float t = w * g.rcp;
    float r = (t + 12582912.0f) - 12582912.0f;
    if (!(fabsf(t - r) < 0.4999f && fabsf(t) < 256.0f)) r = rintf(w / g.scale);
    return r;
}
__device__ __forceinline__ uint32_t code_of(float w, const GroupParams &g) {
    return (uint32_t)(int)fminf(fmaxf(round_quotient(w, g) + g.zero, 0.0f), 15.0f);
}
__device__ __forceinline__ uint32_t codes4(const float (&v)[4], const GroupParams &g) {
    return code_of(v[0], g) | code_of(v[1], g) << 8 | code_of(v[2], g) << 16 | code_of(v[3], g) << 24;
}

// Groups of 128: a warp holds a group in registers, four values per lane, and works on four rows at once. A block covers
// 32 rows of one group column, so that scales and zeros [G, N] leave as whole sectors.
template <int DT, bool SYM>
__global__ void __launch_bounds__(256) quantize128_kernel(const void *__restrict__ w, int64_t N, int64_t K,
                                                          uint32_t *__restrict__ codes, uint16_t *__restrict__ scales,
                                                          int scale_dtype, int8_t *__restrict__ zeros) {
    __shared__ uint16_t s_scale[32];
    __shared__ int8_t s_zero[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gi = blockIdx.x;
    const int64_t n0 = (int64_t)blockIdx.y * 32;
    float v[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int64_t n = n0 + warp * 4 + r;
        if (n < N) load4<DT>(w, n * K + gi * 128 + lane * 4, v[r]);
        else v[r][0] = v[r][1] = v[r][2] = v[r][3] = 0.f;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float lo = min_nan(min_nan(v[r][0], v[r][1]), min_nan(v[r][2], v[r][3]));
        float hi = max_nan(max_nan(v[r][0], v[r][1]), max_nan(v[r][2], v[r][3]));
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo = min_nan(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max_nan(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const GroupParams g = group_params<SYM>(lo, hi, scale_dtype);
        const int64_t n = n0 + warp * 4 + r;
        if (n < N) codes[(n * K + gi * 128) / 4 + lane] = codes4(v[r], g);
        if (lane == 0) {
            s_scale[warp * 4 + r] = g.scale_bits;
            s_zero[warp * 4 + r] = (int8_t)(int)g.zero;
        }
    }
    __syncthreads();
    const int64_t n = n0 + threadIdx.x;
    if (threadIdx.x < 32 && n < N) {
        scales[gi * N + n] = s_scale[threadIdx.x];
        if (!SYM) zeros[gi * N + n] = s_zero[threadIdx.x];
    }
}

// Any group size that is a multiple of 4: a block per (row, group), two passes over the group (the second one reads it
// from L1 or L2).
template <int DT, bool SYM>
__global__ void __launch_bounds__(256) quantize_group_kernel(const void *__restrict__ w, int64_t N, int64_t K, int group,
                                                             uint32_t *__restrict__ codes, uint16_t *__restrict__ scales,
                                                             int scale_dtype, int8_t *__restrict__ zeros) {
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
static void quantize_launch(const void *w, int64_t N, int64_t K, int group, uint32_t *codes, uint16_t *scales,
                            int scale_dtype, int8_t *zeros, cudaStream_t s) {
    if (group == 128 && (N + 31) / 32 <= 65535) {
        const dim3 grid((unsigned)(K / 128), (unsigned)((N + 31) / 32));
        quantize128_kernel<DT, SYM><<<grid, 256, 0, s>>>(w, N, K, codes, scales, scale_dtype, zeros);
    } else {
        const int threads = group >= 1024 ? 256 : group >= 512 ? 128 : group >= 256 ? 64 : 32;
        quantize_group_kernel<DT, SYM><<<(unsigned)(N * (K / group)), threads, 0, s>>>(w, N, K, group, codes, scales,
                                                                                     scale_dtype, zeros);
    }
}

int launch_quantize(qf_ctx *ctx, const void *w, int dtype, int64_t N, int64_t K, int group, bool symmetric, void *codes,
                    void *scales, int scale_dtype, void *zeros, cudaStream_t s) {
    auto *fn = dtype == QF_F16    ? (symmetric ? quantize_launch<QF_F16, true> : quantize_launch<QF_F16, false>)
               : dtype == QF_BF16 ? (symmetric ? quantize_launch<QF_BF16, true> : quantize_launch<QF_BF16, false>)
                                  : (symmetric ? quantize_launch<QF_F32, true> : quantize_launch<QF_F32, false>);
    fn(w, N, K, group, (uint32_t *)codes, (uint16_t *)scales, scale_dtype, (int8_t *)zeros, s);
    g_launch_count.fetch_add(1);
    QF_CUDA_TRY(ctx, cudaGetLastError());
    return QF_OK;
}

}  // namespace qf
