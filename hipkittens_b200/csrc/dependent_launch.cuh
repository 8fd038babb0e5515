// Host side of the dependent launches that ptx::grid_dep_wait and grid_dep_launch describe.
#pragma once

#include <cuda_runtime.h>

namespace hk {

// `early`: launch with programmatic stream serialization, so that the grid may start under the tail of the kernel before it
// in the stream; the kernel has to execute grid_dep_wait in every thread before it touches global memory or leaves.
// Otherwise an ordinary launch, which starts when everything before it has completed.
template <typename... Params, typename... Args>
cudaError_t launch_dependent(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace hk
