// Host side of the tensor-map helpers (see tma.cuh).
#include "tma.cuh"
#include "common.cuh"
#include <mutex>
#include <unordered_map>

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool looked = false;
    if (!looked) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        looked = true;
    }
    return fn;
}

static int encode_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes,
                     uint32_t box_rows, uint32_t box_cols, int swizzle, CUtensorMapDataType type, uint32_t size) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        dl_fail(DL_ERR_LAUNCH, "tensor map: the driver offers no cuTensorMapEncodeTiled");
        return -1;
    }
    if (((uintptr_t)base % 16) || (pitch_bytes % 16) || ((box_cols * size) % 16) || box_rows > 256 || box_cols > 256 ||
        (swizzle == DL_TMAP_SWIZZLE_128B && box_cols * size != 128) || (swizzle == DL_TMAP_SWIZZLE_64B && box_cols * size != 64)) {
        dl_fail(DL_ERR_ARGUMENT, "tensor map: base %p pitch %llu box %ux%u swizzle %d break the alignment rules", base,
                (unsigned long long)pitch_bytes, box_rows, box_cols, swizzle);
        return -2;
    }
    const cuuint64_t dims[2] = {cols, rows};                  // innermost first
    const cuuint64_t strides[1] = {pitch_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(out, type, 2, const_cast<void*>(base), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swizzle == DL_TMAP_SWIZZLE_128B  ? CU_TENSOR_MAP_SWIZZLE_128B
                          : swizzle == DL_TMAP_SWIZZLE_64B ? CU_TENSOR_MAP_SWIZZLE_64B
                                                           : CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        dl_fail(DL_ERR_LAUNCH, "tensor map: cuTensorMapEncodeTiled returned %d (rows %llu cols %llu pitch %llu box %ux%u)",
                (int)r, (unsigned long long)rows, (unsigned long long)cols, (unsigned long long)pitch_bytes, box_rows, box_cols);
        return -2;
    }
    return 0;
}

int dl_tmap_encode_2d_bf16(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes,
                           uint32_t box_rows, uint32_t box_cols, int swizzle) {
    return encode_2d(out, base, rows, cols, pitch_bytes, box_rows, box_cols, swizzle, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
}

namespace {
struct MapKey {
    const void* base;
    unsigned long long rows, cols, pitch;
    uint32_t box_rows, box_cols;
    int swizzle, f32;
    bool operator==(const MapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && pitch == o.pitch && box_rows == o.box_rows &&
               box_cols == o.box_cols && swizzle == o.swizzle && f32 == o.f32;
    }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        size_t h = std::hash<const void*>()(k.base);
        h = h * 1000003u ^ (size_t)k.rows;
        h = h * 1000003u ^ (size_t)k.cols;
        h = h * 1000003u ^ (size_t)k.pitch;
        h = h * 1000003u ^ ((size_t)k.box_rows << 20 | (size_t)k.box_cols << 4 | (size_t)k.swizzle << 1 | (size_t)k.f32);
        return h;
    }
};
}  // namespace

static int cached_2d(CUtensorMap* out, const void* base, unsigned long long rows, unsigned long long cols,
                     unsigned long long pitch_bytes, uint32_t box_rows, uint32_t box_cols, int swizzle, int f32) {
    static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> maps;
    static std::mutex maps_mutex;
    std::lock_guard<std::mutex> lock(maps_mutex);
    const MapKey key{base, rows, cols, pitch_bytes, box_rows, box_cols, swizzle, f32};
    auto it = maps.find(key);
    if (it == maps.end()) {
        CUtensorMap fresh;
        const int rc = encode_2d(&fresh, base, rows, cols, pitch_bytes, box_rows, box_cols, swizzle,
                                 f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, f32 ? 4 : 2);
        if (rc != 0) return rc;
        if (maps.size() > 8192) maps.clear();
        it = maps.emplace(key, fresh).first;
    }
    *out = it->second;
    return 0;
}

int dl_tmap_cached_2d_bf16(CUtensorMap* out, const void* base, unsigned long long rows, unsigned long long cols,
                           unsigned long long pitch_bytes, uint32_t box_rows, uint32_t box_cols, int swizzle) {
    return cached_2d(out, base, rows, cols, pitch_bytes, box_rows, box_cols, swizzle, 0);
}
int dl_tmap_cached_2d_f32(CUtensorMap* out, const void* base, unsigned long long rows, unsigned long long cols,
                          unsigned long long pitch_bytes, uint32_t box_rows, uint32_t box_cols, int swizzle) {
    return cached_2d(out, base, rows, cols, pitch_bytes, box_rows, box_cols, swizzle, 1);
}
