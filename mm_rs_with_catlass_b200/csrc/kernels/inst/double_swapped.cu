// Instantiates the double-tile kernel with swapped roles: features along the tiles' rows, tokens along their columns (see
// double_tile.cuh).
#include "catcoc/double_inst.cuh"

namespace catcoc { namespace inst {
cudaError_t prepare_double_swapped() {
  const cudaError_t e = set_swapped_attrs<KIND_F16>();
  return e == cudaSuccess ? set_swapped_attrs<KIND_I8>() : e;
}
cudaError_t prepare_double() {
  cudaError_t e = prepare_double_f16();
  if (e == cudaSuccess) e = prepare_double_8bit();
  return e == cudaSuccess ? prepare_double_swapped() : e;
}
cudaError_t launch_double(int kind, bool full, const FusedParams& p, int grid, cudaStream_t s) {
  if (p.dt.swap == 0) return kind == KIND_F16 ? launch_double_f16(full, p, grid, s) : launch_double_8bit(kind, full, p, grid, s);
  if (kind == KIND_F16) return launch_double_swapped<KIND_F16>(full, p, grid, s);
  return kind == KIND_I8 ? launch_double_swapped<KIND_I8>(full, p, grid, s) : cudaErrorNotSupported;
}
cudaError_t launch_double_tokens(int kind, bool full, const FusedParamsTok& p, int grid, cudaStream_t s) {
  if (kind == KIND_F16) return launch_double_swapped<KIND_F16>(full, p, grid, s);
  return kind == KIND_I8 ? launch_double_swapped<KIND_I8>(full, p, grid, s) : cudaErrorNotSupported;
}
} }
