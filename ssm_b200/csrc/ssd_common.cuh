// What the tensor-core kernels of the state-space-dual scan share: tile sizes and the tensor maps of their operands.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tc05.cuh"

namespace ssmb {

constexpr int kQ = 256;    // chunk length
constexpr int kP = 64;     // head dimension
constexpr int kN = 128;    // state dimension
constexpr int kBlk = 128;  // rows per CTA of the per-chunk kernels

// cuTensorMapEncodeTiled, fetched through the runtime: no link-time dependency on the driver
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}
// (batch, len, outer, inner) tensor of 16-bit elements seen as rank 4 (inner, outer, step, batch);
// box = 64 inner elements of one outer index x `rows` steps
inline int encode_rows_map(CUtensorMap* m, const void* base, int batch, int len, int outer, int inner, int rows, int io_dtype) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return ::ssmb::fail(SSM_ERR_DEVICE, "ssd_scan: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)len, (cuuint64_t)batch};
  const cuuint64_t strides[3] = {(cuuint64_t)inner * 2, (cuuint64_t)outer * inner * 2, (cuuint64_t)len * outer * inner * 2};
  const cuuint32_t box[4] = {(cuuint32_t)kP, 1, (cuuint32_t)rows, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = io_dtype == SSM_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const CUresult rc = fn(m, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return ::ssmb::fail(SSM_ERR_DEVICE, "ssd_scan: cuTensorMapEncodeTiled rejected the tensor");
  return SSM_OK;
}

}  // namespace ssmb
