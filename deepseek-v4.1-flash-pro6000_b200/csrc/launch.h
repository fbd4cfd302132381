// Programmatic dependent launch: the kernel's launch and prologue overlap the end of the kernel in front of it in the
// stream.  Every kernel launched this way calls cudaGridDependencySynchronize() before it touches global memory, in every
// CTA and on every path, so that the completion of a kernel still implies that of everything in front of it.
#pragma once
#include <cuda_runtime.h>

namespace ds41 {

inline cudaLaunchAttribute programmatic_launch() {
  cudaLaunchAttribute a{};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

}  // namespace ds41
