// Programmatic dependent launch: the kernel's launch and prologue overlap the end of the kernel in front of it in the
// stream.  Every kernel launched this way calls cudaGridDependencySynchronize() in every CTA, on every path, before it touches
// what an earlier kernel may have written, and lets the kernel behind it start only after that call; so when a kernel
// starts early, everything in front of its predecessor has finished, and weights, which no kernel of this library writes,
// may be read before the call.
#pragma once
#include <cuda_runtime.h>

namespace ds41 {

inline cudaLaunchAttribute programmatic_launch() {
  cudaLaunchAttribute a{};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

template <class... Params, class... Args>
cudaError_t launch_early(void (*kernel)(Params...), int ctas, int threads, size_t smem, cudaStream_t stream, const Args &...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(ctas));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1] = {programmatic_launch()};
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace ds41
