// Programmatic dependent launch: a kernel launched with launch_pdl may start while the kernel
// before it on the stream is still draining, so its launch latency is hidden.  Such a kernel calls
// pdl_wait() before it touches memory that any earlier kernel writes or reads (it returns when
// the kernels before it have finished and their writes are visible); a kernel calls pdl_trigger()
// when the next one may start.  Both do nothing in a plain launch.
#pragma once

#include <cuda_runtime.h>

namespace annc {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline cudaLaunchAttribute pdl_attribute() {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1] = {pdl_attribute()};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace annc
