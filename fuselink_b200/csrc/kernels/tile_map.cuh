// Tensor maps of row-major matrices of 16-bit elements, for TMA loads of 64-column tiles (host side).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace fl {

typedef CUresult (*TileEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline TileEncodeFn tile_encode() {
  static const TileEncodeFn fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) sym = nullptr;
    return reinterpret_cast<TileEncodeFn>(sym);
  }();
  return fn;
}

// [outer, inner] of 16-bit elements (type: CUtensorMapDataType) in boxes of box_outer x 64, 128-byte swizzle; what lies outside is
// read as zeros.  base: a multiple of 16 bytes, inner: of 8.
inline int tile_map(CUtensorMap* m, int type, const void* base, long long inner, long long outer, int box_outer) {
  const TileEncodeFn enc = tile_encode();
  if (enc == nullptr) return -10;
  const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer}, strides[1] = {(cuuint64_t)inner * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_outer}, step[2] = {1, 1};
  return enc(m, (CUtensorMapDataType)type, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -12;
}

}  // namespace fl
