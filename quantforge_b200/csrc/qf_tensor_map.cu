// Tensor maps of the tcgen05 kernels, encoded by the driver once per (address, shape, box) and kept.
#include <mutex>
#include <unordered_map>

#include "qf_tcgen05.cuh"

namespace qf {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;
static std::once_flag g_encode_once;

static EncodeTiledFn get_encode() {
    std::call_once(g_encode_once, [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            g_encode = (EncodeTiledFn)fn;
    });
    return g_encode;
}

struct MapKey {
    const void *ptr;
    uint64_t d0, d1;
    uint32_t b0, b1;
    int kind;  // of get_tensor_map * 8 + swizzle; 2 * 8 + swizzle: a slab
    bool operator==(const MapKey &o) const {
        return ptr == o.ptr && d0 == o.d0 && d1 == o.d1 && b0 == o.b0 && b1 == o.b1 && kind == o.kind;
    }
};
struct MapKeyHash {
    size_t operator()(const MapKey &k) const {
        size_t h = std::hash<const void *>()(k.ptr);
        h ^= std::hash<uint64_t>()(k.d0 * 1000003u + k.d1) + 0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2);
        h ^= std::hash<uint64_t>()(((uint64_t)k.b0 << 32) | k.b1 | ((uint64_t)k.kind << 60)) + (h << 6) + (h >> 2);
        return h;
    }
};
static std::mutex g_map_mutex;
static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_maps;

static bool known_map(const MapKey &key, CUtensorMap *out) {
    std::lock_guard<std::mutex> g(g_map_mutex);
    const auto itf = g_maps.find(key);
    if (itf == g_maps.end()) return false;
    *out = itf->second;
    return true;
}

static int encode_map(qf_ctx *ctx, const MapKey &key, CUtensorMap *out, CUtensorMapDataType type, cuuint32_t rank,
                      const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box, CUtensorMapSwizzle swz) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return fail(ctx, QF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(out, type, rank, const_cast<void *>(key.ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, QF_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    std::lock_guard<std::mutex> g(g_map_mutex);
    if (g_maps.size() > 4096) g_maps.clear();
    g_maps[key] = *out;
    return QF_OK;
}

int get_tensor_map(qf_ctx *ctx, CUtensorMap *out, const void *ptr, int kind, uint64_t inner, uint64_t outer, uint32_t box_inner,
                   uint32_t box_outer, CUtensorMapSwizzle swz) {
    const MapKey key{ptr, inner, outer, box_inner, box_outer, kind * 8 + (int)swz};
    if (known_map(key, out)) return QF_OK;
    const cuuint64_t dims[2] = {inner, outer}, strides[1] = {inner * (kind == 0 ? 1 : 2)};
    const cuuint32_t box[2] = {box_inner, box_outer};
    return encode_map(ctx, key, out, kind == 0 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, dims, strides, box,
                      swz);
}

int get_slab_map(qf_ctx *ctx, CUtensorMap *out, const void *blob, uint64_t blocks, uint64_t chunks) {
    constexpr uint64_t kLines = QF_SLAB_UNIT_BYTES / 64;
    const MapKey key{blob, blocks, chunks, 64, 2, 2 * 8 + (int)CU_TENSOR_MAP_SWIZZLE_64B};
    if (known_map(key, out)) return QF_OK;
    const cuuint64_t dims[4] = {64, kLines, chunks, blocks}, strides[3] = {64, kLines * 64, chunks * kLines * 64};
    const cuuint32_t box[4] = {64, (cuuint32_t)kLines, 1, 2};
    return encode_map(ctx, key, out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}

}  // namespace qf
