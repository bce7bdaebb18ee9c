#pragma once

#include "common.cuh"

namespace kb2::dev {

// The K-cycle's scalar steps (scalars.kern.h:154-186), each run by one thread of
// the reduction that produces its operands: as kernels of one thread they cost a
// launch of 1.1 us each, four times per inner step.
__device__ __forceinline__ void inner_alpha(float* scalars, int* status, bool first) {
  const Pair denom = kp_load(scalars, 0);
  const Pair alpha = kp_div(kp_load(scalars, 2), denom);
  if (!kp_positive(denom) || !kp_coefficient(alpha) ||
      (kp_zero(alpha) && !kp_zero(kp_load(scalars, 2))))
    status[0] = first ? 2 : 1;
  else
    kp_store(scalars, 8, alpha);
}
// Adaptive exit: keep the first correction when |t|^2 <= |b|^2 / 16.
__device__ __forceinline__ void inner_check(const float* scalars, int* status) {
  if (kp_le(kp_load(scalars, 4), kp_mul(kp(0.0625f, 0.0f), kp_load(scalars, 6)))) status[0] = 1;
}
__device__ __forceinline__ void inner_beta(float* scalars, int* status) {
  const Pair beta = kp_div(kp_neg(kp_load(scalars, 4)), kp_load(scalars, 0));
  if (!kp_coefficient(beta) || (kp_zero(beta) && !kp_zero(kp_load(scalars, 4))))
    status[0] = 1;
  else
    kp_store(scalars, 10, beta);
}

}  // namespace kb2::dev
