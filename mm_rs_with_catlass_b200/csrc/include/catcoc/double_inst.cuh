// Launch helpers of the double-tile kernel, shared by its instantiation units (kernels/inst/double_*.cu).
#pragma once
#include <cstring>

#include "catcoc/double_tile.cuh"
#include "catcoc/kernel_inst.cuh"

namespace catcoc {
namespace inst {

template <int KIND, bool FULL, bool SWAP, class Params>
cudaError_t set_double_attr() {
  return cudaFuncSetAttribute(dtile::double_tile_kernel<KIND, FULL, SWAP, Params>, cudaFuncAttributeMaxDynamicSharedMemorySize, dtile::kSmemBytes);
}

template <int KIND, bool FULL, bool SWAP, class Params>
cudaError_t launch_double_one(const Params& p, int grid, cudaStream_t stream) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(dtile::kThreads, 1, 1);
  cfg.dynamicSmemBytes = dtile::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  // set up while its predecessor in the stream drains (see host::launch_overlapped)
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, dtile::double_tile_kernel<KIND, FULL, SWAP, Params>, p);
}

// the epilogue variant that a launch needs
template <int KIND, class Params>
cudaError_t launch_double_swapped(bool full, const Params& p, int grid, cudaStream_t s) {
  return full ? launch_double_one<KIND, true, true>(p, grid, s) : launch_double_one<KIND, false, true>(p, grid, s);
}
template <int KIND>
cudaError_t set_double_attrs() {
  cudaError_t e = set_double_attr<KIND, false, false, FusedParams>();
  if (e == cudaSuccess) e = set_double_attr<KIND, true, false, FusedParams>();
  return e;
}
template <int KIND>
cudaError_t set_swapped_attrs() {
  cudaError_t e = set_double_attr<KIND, false, true, FusedParams>();
  if (e == cudaSuccess) e = set_double_attr<KIND, true, true, FusedParams>();
  if (e == cudaSuccess) e = set_double_attr<KIND, false, true, FusedParamsTok>();
  if (e == cudaSuccess) e = set_double_attr<KIND, true, true, FusedParamsTok>();
  return e;
}

cudaError_t prepare_double_f16();
cudaError_t prepare_double_8bit();
cudaError_t prepare_double_swapped();

}  // namespace inst
}  // namespace catcoc
