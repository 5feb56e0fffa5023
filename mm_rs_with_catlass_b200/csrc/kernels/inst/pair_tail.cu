// Instantiates the fused kernel for local products on pair tiles whose last tiles are cut along K (see FusedParamsTail).
#include "catcoc/kernel_inst.cuh"

namespace catcoc { namespace inst {
cudaError_t prepare_tail() {
  cudaError_t e = set_smem_attr<KIND_F16, true, EPI_PLAIN, FusedParamsTail>();
  if (e == cudaSuccess) e = set_smem_attr<KIND_F16, true, EPI_FULL, FusedParamsTail>();
  if (e == cudaSuccess) e = set_smem_attr<KIND_I8, true, EPI_PLAIN, FusedParamsTail>();
  if (e == cudaSuccess) e = set_smem_attr<KIND_I8, true, EPI_FULL, FusedParamsTail>();
  return e;
}
cudaError_t launch_tail(int kind, bool full, const FusedParamsTail& p, int grid, cudaStream_t s) {
  if (kind == KIND_F16)
    return full ? launch_one<KIND_F16, true, EPI_FULL>(p, grid, 0, s) : launch_one<KIND_F16, true, EPI_PLAIN>(p, grid, 0, s);
  if (kind == KIND_I8)
    return full ? launch_one<KIND_I8, true, EPI_FULL>(p, grid, 0, s) : launch_one<KIND_I8, true, EPI_PLAIN>(p, grid, 0, s);
  return cudaErrorNotSupported;
}
} }
