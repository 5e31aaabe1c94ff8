// Host side of the TMA descriptions in weight_maps.h.  cuTensorMapEncodeTiled is a pure host function
// fetched from the driver at run time (no link against libcuda).
#include <atomic>

#include "common.cuh"
#include "weight_maps.h"

namespace mlxr {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int tensor_map_encoder(EncodeTiledFn* out) {
  static std::atomic<EncodeTiledFn> encode{nullptr};
  EncodeTiledFn e = encode.load(std::memory_order_acquire);
  if (!e) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    MLXR_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    if (!fn || q != cudaDriverEntryPointSuccess) { set_error("cuTensorMapEncodeTiled is not available in this driver"); return MLXR_ERR_CUDA; }
    e = (EncodeTiledFn)fn;
    encode.store(e, std::memory_order_release);
  }
  *out = e;
  return MLXR_OK;
}

int device_sms(int* out) {
  static std::atomic<int> sms[64];
  int dev = 0;
  MLXR_CUDA_TRY(cudaGetDevice(&dev));
  int n = sms[dev & 63].load();
  if (!n) {
    MLXR_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    sms[dev & 63].store(n);
  }
  *out = n;
  return MLXR_OK;
}

static int encode_2d(CUtensorMapDataType type, const void* base, size_t cols, size_t rows, size_t stride, int box_cols, int box_rows,
                     CUtensorMapSwizzle swizzle, CUtensorMap* out) {
  EncodeTiledFn encode = nullptr;
  if (int r = tensor_map_encoder(&encode)) return r;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)stride};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(out, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d) for %zu rows of %zu bytes", (int)r, rows, stride); return MLXR_ERR_CUDA; }
  return MLXR_OK;
}

int weight_maps(int qt, const void* w, int N, int K, int tile_rows, CUtensorMap* out, int* odd_shift) {
  // packed rows as 8-byte elements
  if (qt != MLXR_NF4) {
    const int unit = qt == MLXR_Q8_0 ? 272 : 144;
    const size_t rb = (size_t)(K / 256) * unit;
    return encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT64, w, rb / 8, N, rb, unit / 8, tile_rows, CU_TENSOR_MAP_SWIZZLE_NONE, out);
  }
  const size_t rb = (size_t)(K / 256) * 136;
  const int sh = (int)(rb & 8);
  *odd_shift = sh;
  if (int r = encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT64, w, rb / 8, (N + 1) / 2, 2 * rb, 18, tile_rows / 2, CU_TENSOR_MAP_SWIZZLE_NONE, out)) return r;
  return encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT64, (const char*)w + rb - sh, (rb + sh) / 8, N / 2, 2 * rb, 18, tile_rows / 2, CU_TENSOR_MAP_SWIZZLE_NONE, out + 1);
}

int rows_map(const void* w, int rows, size_t row_bytes, int box_bytes, int box_rows, CUtensorMap* out) {
  return encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT64, w, row_bytes / 8, rows, row_bytes, box_bytes / 8, box_rows, CU_TENSOR_MAP_SWIZZLE_NONE, out);
}

int activation_map(const void* x, int M, int K, int dtype, int rows, CUtensorMap* out) {
  return encode_2d(dtype == MLXR_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, K, M, (size_t)K * 2, 64, rows,
                   CU_TENSOR_MAP_SWIZZLE_128B, out);
}

int activation_blocks_map(const void* x, int M, int K, int dtype, int rows, int blocks, CUtensorMap* out) {
  EncodeTiledFn encode = nullptr;
  if (int r = tensor_map_encoder(&encode)) return r;
  const cuuint64_t dims[3] = {64, (cuuint64_t)M, (cuuint64_t)(K / 64)}, strides[2] = {(cuuint64_t)K * 2, 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)rows, (cuuint32_t)blocks}, estr[3] = {1, 1, 1};
  const CUresult r = encode(out, dtype == MLXR_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(x), dims, strides, box,
                            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d) for X [%d, %d]", (int)r, M, K); return MLXR_ERR_CUDA; }
  return MLXR_OK;
}

int result_map(void* y, int M, int N, int dtype, int box_cols, int box_rows, CUtensorMap* out) {
  return encode_2d(dtype == MLXR_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, y, N, M, (size_t)N * 2, box_cols, box_rows,
                   box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE, out);
}

}  // namespace mlxr
