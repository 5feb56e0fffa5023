// Instantiates the double-tile kernel for 16-bit operands (see double_tile.cuh).
#include "catcoc/double_inst.cuh"

namespace catcoc { namespace inst {
cudaError_t prepare_double_f16() {
  const cudaError_t e = set_double_attrs<KIND_F16>();
  return e == cudaSuccess ? set_double_attr<KIND_F16, false, false, FusedParamsGk>() : e;
}
cudaError_t launch_double_f16(bool full, const FusedParams& p, int grid, cudaStream_t s) {
  return full ? launch_double_one<KIND_F16, true, false>(p, grid, s) : launch_double_one<KIND_F16, false, false>(p, grid, s);
}
cudaError_t launch_double_slice_k(const FusedParamsGk& p, int grid, cudaStream_t s) { return launch_double_one<KIND_F16, false, false>(p, grid, s); }
} }
