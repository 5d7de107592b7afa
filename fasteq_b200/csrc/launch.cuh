// Launch of a kernel that calls wait_for_previous_kernel(): it may begin before the kernel ahead of it in the stream has ended, so that its
// launch and set-up (barriers, tensor memory, descriptors: 1 to 2 us) lie beside the other's tail.  Only for kernels that write global
// memory after that wait alone.  Ahead of it they read only what was complete before the kernel ahead could begin (a graph's plan); the rest
// after it, in a way no compiler can move ahead of it: bulk and tensor copies, loads whose addresses depend on those, volatile
// loads, plain ones through pointers without __restrict__.  Captured into CUDA graphs as programmatic edges.
#pragma once
#include <cuda_runtime.h>

namespace fasteq {

template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace fasteq
