// Instantiates the fused kernel for 16-bit products over ragged K ranges (see FusedParamsGk).
#include "catcoc/kernel_inst.cuh"

namespace catcoc { namespace inst {
cudaError_t prepare_slice_k() {
  const cudaError_t e = set_smem_attr<KIND_F16, false, EPI_PLAIN, FusedParamsGk>();
  return e == cudaSuccess ? set_smem_attr<KIND_F16, true, EPI_PLAIN, FusedParamsGk>() : e;
}
cudaError_t launch_slice_k(bool pair, const FusedParamsGk& p, int grid, cudaStream_t s) {
  return pair ? launch_one<KIND_F16, true, EPI_PLAIN>(p, grid, 0, s) : launch_one<KIND_F16, false, EPI_PLAIN>(p, grid, 0, s);
}
} }
