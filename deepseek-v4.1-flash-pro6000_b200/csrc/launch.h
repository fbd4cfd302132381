// Programmatic dependent launch: the kernel's launch and prologue overlap the end of the kernel in front of it in the
// stream.  Every kernel launched this way calls cudaGridDependencySynchronize() in every CTA, on every path, before it reads or
// writes anything that another kernel may write or read.  That includes the weights: the kernel in front may be the one that
// writes them, and may let its successor start long before it has finished.  What comes earlier is set-up on chip and, for the
// weights, prefetch_l2: a line on its way into the L2 is a copy that later writes replace there, so it hides the memory's
// latency without fixing what will be read.
// Since every kernel waits for the one in front of it to have finished, which waited likewise, everything in front of a kernel has
// finished once its own wait returns, whenever each of them let its successor start: most do so right after their wait, the
// kernel that clears the head's records before it, the last of a call not at all (its end does).
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

// Loads of such data go this way (or are plain): the read-only path (__ldg, const __restrict__ parameters) is only for what nobody
// writes while the kernel runs, and an early kernel runs while the one in front still writes.
template <class T>
__device__ __forceinline__ T load_input(const T *p) { return __ldca(p); }

__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
}

}  // namespace ds41
