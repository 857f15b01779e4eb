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
cudaError_t pdl_launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace pthb200
