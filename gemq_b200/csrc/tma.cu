// Cached cuTensorMapEncodeTiled for 2-D row-major tensors (driver entry point resolved at run
// time, so the library has no link-time dependency on libcuda).
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"

namespace gemq {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

struct MapKey {
  const void* base;
  long long rows;
  int inner, elem, box_inner, box_rows, swz, dev;
  bool operator<(const MapKey& o) const {
    return std::tie(base, rows, inner, elem, box_inner, box_rows, swz, dev) <
           std::tie(o.base, o.rows, o.inner, o.elem, o.box_inner, o.box_rows, o.swz, o.dev);
  }
};

// elem_bytes 4 -> UINT32, 2 -> UINT16 (any 16-bit type).  `inner` elements per row, row stride
// inner * elem_bytes (a multiple of 16).  128B swizzle needs box_inner * elem_bytes <= 128.
static std::mutex g_mu;
static std::map<MapKey, CUtensorMap> g_cache;

bool tensor_map_2d(CUtensorMap* out, const void* base, int elem_bytes, int inner, long long rows, int box_inner,
                   int box_rows, bool swizzle128) {
  int dev = 0;
  cudaGetDevice(&dev);
  const MapKey key{base, rows, inner, elem_bytes, box_inner, box_rows, swizzle128 ? 1 : 0, dev};
  std::lock_guard<std::mutex> lock(g_mu);
  auto it = g_cache.find(key);
  if (it != g_cache.end()) {
    *out = it->second;
    return true;
  }
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(inner) * elem_bytes};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_inner), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1u, 1u};
  CUtensorMap m;
  const CUresult r = enc(&m, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return false;
  if (g_cache.size() > 4096) g_cache.clear();
  g_cache[key] = m;
  *out = m;
  return true;
}

// 3-D view (32 columns, rows, strips): one box brings `strips` neighbouring 32-column strips of 16 rows,
// each as 16 swizzled rows of 128 bytes.  One such instruction replaces a 2-D box per strip: a warp's
// lanes issue their boxes one after the other, about 50 cycles each.
bool tensor_map_strips(CUtensorMap* out, const void* base, int N, long long rows, int strips) {
  int dev = 0;
  cudaGetDevice(&dev);
  const MapKey key{base, rows, N, 4, 32, 16, 16 + strips, dev};
  std::lock_guard<std::mutex> lock(g_mu);
  auto it = g_cache.find(key);
  if (it != g_cache.end()) {
    *out = it->second;
    return true;
  }
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {32, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(N / 32)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(N) * 4, 128};
  const cuuint32_t box[3] = {32, 16, static_cast<cuuint32_t>(strips)};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  CUtensorMap m;
  if (enc(&m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(base), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (g_cache.size() > 4096) g_cache.clear();
  g_cache[key] = m;
  *out = m;
  return true;
}

// 16-bit activations [rows, K] as (64, rows, K / 64): one box brings `box_rows` rows of two neighbouring 64-wide
// k-blocks, each as swizzled rows of 128 bytes; a block past the end is zero-filled.
bool tensor_map_blocks(CUtensorMap* out, const void* base, int K, long long rows, int box_rows) {
  int dev = 0;
  cudaGetDevice(&dev);
  const MapKey key{base, rows, K, 2, 64, box_rows, 2, dev};
  std::lock_guard<std::mutex> lock(g_mu);
  auto it = g_cache.find(key);
  if (it != g_cache.end()) {
    *out = it->second;
    return true;
  }
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(K / 64)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(K) * 2, 128};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 2};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  CUtensorMap m;
  if (enc(&m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (g_cache.size() > 4096) g_cache.clear();
  g_cache[key] = m;
  *out = m;
  return true;
}

}  // namespace gemq
