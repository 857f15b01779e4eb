// Programmatic dependent launch: a kernel launched with pdl_launch may start while the kernel in front of it in
// the stream still runs, as soon as every CTA of that one has called pdl_trigger or left.  It calls pdl_wait, in every
// CTA and before it leaves, ahead of the first access to anything that earlier work writes or reads: the wait returns
// when the kernel in front is complete and its writes are visible.  (A kernel in front that never triggers is waited for
// as without this.)
#pragma once

#include <cuda_runtime.h>

namespace pthb200 {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... Params, class... Args>
cudaError_t pdl_launch_clusters(int cluster, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  return err != cudaSuccess ? err : cudaGetLastError();
}
template <class... Params, class... Args>
cudaError_t pdl_launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  return pdl_launch_clusters(1, kernel, grid, block, smem, stream, static_cast<Args&&>(args)...);
}

}  // namespace pthb200
