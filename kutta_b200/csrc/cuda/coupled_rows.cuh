// Block arithmetic shared by the Coupled solve's fine and coarse kernels
// (compiled with --fmad=false): the reference's operations in their order.
#pragma once

#include "common.cuh"

namespace kb2::dev {

// Neumaier-compensated sum (fv_coupled.kern.h:77-84).
struct Csum {
  float s, e;
};
__device__ __forceinline__ Csum csum_add(Csum a, float b) {
  const float t = a.s + b;
  const float e = fabsf(a.s) >= fabsf(b) ? (a.s - t) + b : (b - t) + a.s;
  return Csum{t, a.e + e};
}
__device__ __forceinline__ float csum_value(Csum a) { return a.s + a.e; }

// The arrow block's inverse (fv_coupled.kern.h:51-60), returned as the five
// factors the block solve uses and the Schur denominator.
struct BlockInverse {
  float iu, iv, iw, hu, hv, hw, schur;
};
__device__ __forceinline__ BlockInverse block_prepare(float du, float dv, float dw, float ex,
                                                      float ey, float ez, float hx, float hy,
                                                      float hz, float c) {
  BlockInverse b;
  b.iu = 1.0f / du;
  b.iv = 1.0f / dv;
  b.iw = 1.0f / dw;
  b.schur = fmaxf(c - (hx * ex * b.iu + hy * ey * b.iv + hz * ez * b.iw), 0.5f * c);
  b.hu = hx * b.iu;
  b.hv = hy * b.iv;
  b.hw = hz * b.iw;
  return b;
}
// The block solve (fv_coupled.kern.h:61-66).
__device__ __forceinline__ float4 block_solve(float4 r, float ex, float ey, float ez, float iu,
                                              float iv, float iw, float hu, float hv, float hw,
                                              float schur) {
  const float p = (r.w - hu * r.x - hv * r.y - hw * r.z) / schur;
  return make_float4(iu * (r.x - ex * p), iv * (r.y - ey * p), iw * (r.z - ez * p), p);
}
// next = base + omega d, base = x, or +0 on a zero start (the reference adds
// the zero explicitly, which turns a -0 step into +0).
__device__ __forceinline__ float4 damped(float4 base, float4 d, float omega) {
  return make_float4(base.x + omega * d.x, base.y + omega * d.y, base.z + omega * d.z,
                     base.w + omega * d.w);
}

}  // namespace kb2::dev
