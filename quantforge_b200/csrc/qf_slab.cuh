// What the kernels that stream QF_LAYOUT_GEMV_SLAB weights through mma.sync share: sizes, shared-memory loads at constant offsets,
// the (value, token) words of partial sums, converter constants and the output store.
#pragma once

#include "qf_common.cuh"
#include "qf_mbar.cuh"

namespace qf {

constexpr int SLAB_THREADS = 160;
constexpr int SLAB_TILE_BYTES = 1088;           // 2 x 512 B of codes + 64 B of constants
constexpr int SLAB_UNIT_BYTES = QF_SLAB_UNIT_BYTES;
constexpr int SLAB_X_PITCH = 576;               // bytes between batch rows of a stage's activation slices (2 x 256 + 64
                                                // of skew: rows g and g+1 land in different shared-memory banks)
constexpr int SLAB_MAX_DEPTH = 16;
static_assert(SLAB_UNIT_BYTES == 4 * SLAB_TILE_BYTES, "unit = 4 tiles");

#ifdef __CUDACC__

// Shared-memory loads with the constant part of the address as an immediate (no address arithmetic in the loop).
template <int OFF>
__device__ __forceinline__ uint32_t lds32_at(uint32_t base) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(base), "n"(OFF));
    return v;
}
template <int OFF>
__device__ __forceinline__ uint4 lds128_at(uint32_t base) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(base), "n"(OFF));
    return v;
}
// Two (value, token) words with one 16-byte access; each 8-byte word is written and read whole.
__device__ __forceinline__ void st_pairs2(unsigned long long *ptr, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(ptr), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_pairs2(const unsigned long long *ptr, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(ptr) : "memory");
}
__device__ __forceinline__ unsigned long long pair_of(float v) {
    return (unsigned long long)__float_as_uint(v) | (1ull << 32);
}

__device__ __forceinline__ float load_out(const void *R, int out_dtype, int64_t idx) {
    if (out_dtype == QF_F32) return reinterpret_cast<const float *>(R)[idx];
    if (out_dtype == QF_F16) return __half2float(reinterpret_cast<const __half *>(R)[idx]);
    return __bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(R)[idx]);
}

template <bool BF16>
__device__ __forceinline__ ZeroScale<BF16> slab_consts(uint32_t word) {
    ZeroScale<BF16> zs;
    // low half / high half broadcast, written as register pack / unpack so that the assembler may fold the
    // broadcast into the operand selectors of the packed-half instructions that consume it
    asm("{.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tmov.b32 %0, {lo, lo};\n\tmov.b32 %1, {hi, hi};}"
        : "=r"(zs.zsub), "=r"(zs.s2)
        : "r"(word));
    // f16 only: -(64 + z) = (1024 + z) * (-1) + 960, exact in f16
    zs.zfma = BF16 ? 0u : fma_f16x2(zs.zsub, 0xbc00bc00u, 0x63806380u);
    return zs;
}

// Writes the finished 16 x M outputs a warp holds for weight rows n0 + {g, g+8} (lane = 4g + t owns batch rows
// nt*8 + 2t + {0, 1}).
template <int MT, typename P>
__device__ __forceinline__ void slab_store(const P &p, int64_t n0, int g, int t, const float (&v)[MT][4]) {
#pragma unroll
    for (int nt = 0; nt < MT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t m = nt * 8 + 2 * t + e;
            if (m >= p.M) continue;
            if (p.epilogue == QF_EPI_SILU_MUL) {
                // rows g of the tile are gate rows, rows g+8 the matching up rows
                const float gate = v[nt][e], up = v[nt][2 + e];
                store_out(p.Y, p.out_dtype, m * (p.N >> 1) + (n0 >> 1) + g, gate / (1.f + expf(-gate)) * up);
            } else {
                const int64_t ia = m * p.N + n0 + g, ib = ia + 8;
                float a = v[nt][e], b = v[nt][2 + e];
                if (p.epilogue == QF_EPI_RESIDUAL_ADD) {
                    a += load_out(p.residual, p.out_dtype, ia);
                    b += load_out(p.residual, p.out_dtype, ib);
                }
                store_out(p.Y, p.out_dtype, ia, a);
                store_out(p.Y, p.out_dtype, ib, b);
            }
        }
}

#endif  // __CUDACC__

}  // namespace qf
