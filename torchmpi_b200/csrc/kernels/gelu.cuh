// GELU (erf form) and its derivative, shared by the elementwise passes (bias_grad.cu) and the GEMM epilogue.
#pragma once
#include <cuda_runtime.h>

namespace tmpi {

// gelu(z) = z * Phi(z);  d/dz [z * Phi(z)] = Phi(z) + z * phi(z).  Phi through the rational erf approximation of Abramowitz and
// Stegun 7.1.26 (absolute error 1.5e-7), which shares its exp(-z^2 / 2) with phi: one ex2, one rcp and a
// dozen FMAs per element keep the kernel memory bound where erff() made it ALU bound.
__device__ __forceinline__ void normal_parts(float z, float* cdf, float* e) {
  *e = __expf(-0.5f * z * z);
  const float t = __fdividef(1.f, fmaf(0.3275911f * 0.70710678118654752f, fabsf(z), 1.f));
  float poly = fmaf(1.061405429f, t, -1.453152027f);
  poly = fmaf(poly, t, 1.421413741f);
  poly = fmaf(poly, t, -0.284496736f);
  poly = fmaf(poly, t, 0.254829592f);
  const float q = 0.5f * poly * t * *e;                 // 1 - Phi(|z|)
  *cdf = z >= 0.f ? 1.f - q : q;
}

__device__ __forceinline__ float gelu_grad(float z) {
  float cdf, e;
  normal_parts(z, &cdf, &e);
  return fmaf(z * 0.3989422804014327f, e, cdf);
}

__device__ __forceinline__ float gelu_value(float z) {
  float cdf, e;
  normal_parts(z, &cdf, &e);
  return z * cdf;
}

}  // namespace tmpi
