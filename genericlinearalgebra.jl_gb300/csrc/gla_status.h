// CUDA errors as statuses of the C ABI (include/glagpu.h).
#pragma once
#include <cuda_runtime.h>

namespace gla {

// -1000 - e. The runtime keeps a failed allocation as the thread's last error,
// and the next launch's check, in a later call that has memory again, would
// report it a second time: it is taken back here.
inline int cuda_status(cudaError_t e) {
  if (e == cudaErrorMemoryAllocation) (void)cudaGetLastError();
  return -1000 - (int)e;
}

}  // namespace gla
