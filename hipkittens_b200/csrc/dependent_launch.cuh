// Host side of the dependent launches that ptx::grid_dep_wait and grid_dep_launch describe.
#pragma once

#include <cuda_runtime.h>

namespace hk {

constexpr int kMaxCluster = 16;  // above 8 a kernel needs cudaFuncAttributeNonPortableClusterSizeAllowed

// CTAs per cluster along x, which divides the grid's x.
struct ClusterX {
  unsigned n;
};

// `early`: launch with programmatic stream serialization, so that the grid may start under the tail of the kernel before it
// in the stream; the kernel has to execute grid_dep_wait in every thread before it touches global memory or leaves.
// Otherwise an ordinary launch, which starts when everything before it has completed.
template <typename... Params, typename... Args>
cudaError_t launch_dependent(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, ClusterX cluster, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (early) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster.n > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster.n;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
cudaError_t launch_dependent(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, const Args&... args) {
  return launch_dependent(early, kernel, grid, block, smem, stream, ClusterX{1}, args...);
}

// Clusters of n CTAs that the current device holds at once (0: not even one, as on a slice of a GPU).
template <typename Kernel>
int clusters_held(Kernel* fn, int threads, size_t smem, int n) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = n;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int held = 0;
  if (cudaOccupancyMaxActiveClusters(&held, fn, &cfg) == cudaSuccess) return held;
  cudaGetLastError();
  return 0;
}

}  // namespace hk
