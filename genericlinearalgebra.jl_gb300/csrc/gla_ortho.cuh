// What the complex and quaternion paths share to bring eigenvectors to working
// orthogonality by Newton-Schulz steps V <- V (I + R/2), R = I - V^H V.
#pragma once
#include <cuda_runtime.h>

namespace gla {

// A step leaves 3/4 R^2. With no entry of R / 2 above 2^-30 that is below
// 3e-16 also for a hundred vectors that are close to one another (their R^2
// has entries up to 100 x 2^-58), so it was the last one. Real eigenvectors
// of groups 32 N u ||A|| apart (N the real order) start with entries of about
// 1/32N: they need three more.
constexpr double kOrthoDone = 0x1p-30;
constexpr int kOrthoSteps = 8;

// The largest of the warp's values (none negative) to *to, as bits.
__device__ __forceinline__ void warp_max_to(double v, unsigned long long* to) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const unsigned long long b = __double_as_longlong(v);
  if ((threadIdx.x & 31) == 0 && b > *(volatile unsigned long long*)to) atomicMax(to, b);
}

}  // namespace gla
