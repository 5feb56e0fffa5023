// Host side shared by the attention kernels: the tensor map of a [batch x heads, sequence, head dimension] operand.
#pragma once
#include "catcoc/capi.h"
#include "catcoc/host_util.h"

namespace catcoc {
namespace host {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [BH, S, D] (D contiguous) as {D, S, BH} with a {64, 128, 1} box: rows past S read as zeros
inline int encode_bsd(CUtensorMap* tm, const void* base, CUtensorMapDataType dt, int64_t BH, int64_t S, int64_t D) {
  static EncodeTiledFn fn = driver_fn<EncodeTiledFn>("cuTensorMapEncodeTiled");
  if (fn == nullptr) return CATCOC_E_DRIVER;
  if (reinterpret_cast<uintptr_t>(base) & 15) { set_error("attention operands must be 16-byte aligned"); return CATCOC_E_ALIGNMENT; }
  cuuint64_t gdim[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(BH)};
  cuuint64_t gstride[2] = {static_cast<cuuint64_t>(D) * 2, static_cast<cuuint64_t>(S) * D * 2};
  cuuint32_t box[3] = {64, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(tm, dt, 3, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (attention) failed: CUresult %d", static_cast<int>(r)); return CATCOC_E_DRIVER; }
  return CATCOC_OK;
}

}  // namespace host
}  // namespace catcoc
