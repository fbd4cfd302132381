// The status words by which a path leaves a row to the kernel behind it in the same call, and what becomes of such a row.
// Plain C++ as well as CUDA, so that a test on the CPU can go through the cases.
#pragma once
#include "ds41_b200.h"

#ifdef __CUDACC__
#define DS41_HOST_DEVICE __host__ __device__
#else
#define DS41_HOST_DEVICE
#endif

namespace ds41 {

// the candidates that were kept may not contain the whole nucleus (of the sharded combine alone it is also a result)
constexpr int kNotCovered = DS41_B200_ROW_NOT_COVERED;
// this path could not certify the row and its nucleus may be wide.  Internal: never returned to the caller
constexpr int kNeedsCluster = -9;

// The row is still the cluster kernel's to decide.
DS41_HOST_DEVICE constexpr bool handed_on(int status) { return status == kNotCovered || status == kNeedsCluster; }

// Status of a row that a cluster no longer reaches because one of its bounded waits expired.  only_handed_on: the launch takes
// only the rows that another path left over, and what that path decided stands.
DS41_HOST_DEVICE constexpr int after_timeout(int status, bool only_handed_on) {
  return only_handed_on && !handed_on(status) ? status : DS41_B200_ROW_TIMEOUT;
}

}  // namespace ds41
