// Instantiates the double-tile kernel for 8-bit operands (see double_tile.cuh).
#include "catcoc/double_inst.cuh"

namespace catcoc { namespace inst {
cudaError_t prepare_double_8bit() {
  cudaError_t e = set_double_attrs<KIND_I8>();
  if (e == cudaSuccess) e = set_double_attrs<KIND_F8>();
  if (e == cudaSuccess) e = set_double_attr<KIND_MX, false, false, FusedParams>();
  return e;
}
cudaError_t launch_double_8bit(int kind, bool full, const FusedParams& p, int grid, cudaStream_t s) {
  if (kind == KIND_I8) return full ? launch_double_one<KIND_I8, true, false>(p, grid, s) : launch_double_one<KIND_I8, false, false>(p, grid, s);
  if (kind == KIND_F8) return full ? launch_double_one<KIND_F8, true, false>(p, grid, s) : launch_double_one<KIND_F8, false, false>(p, grid, s);
  if (kind == KIND_MX && !full) return launch_double_one<KIND_MX, false, false>(p, grid, s);
  return cudaErrorNotSupported;
}
} }
