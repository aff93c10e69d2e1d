// GELU (erf form) and its derivative, shared by the elementwise passes (bias_grad.cu) and the GEMM epilogue.
#pragma once
#include <cuda_runtime.h>
#include "attn_util.cuh"

namespace tmpi {

// gelu(z) = z * Phi(z);  d/dz [z * Phi(z)] = Phi(z) + z * phi(z).  Phi through the rational erf approximation of Abramowitz and
// Stegun 7.1.26 (absolute error 1.5e-7), which shares its exp(-z^2 / 2) with phi: one ex2, one rcp and a
// dozen multiply-adds per element where erff() is a few dozen.  Two elements at a time: the multiply-adds are packed
// fp32 pairs, which halves their issue slots (those bound the GEMM epilogue and the elementwise passes alike), and ex2 and
// rcp flush subnormals (an exponential below 2^-126 adds nothing to either result): the GELU backward with the bias
// gradient, 8192 x 4096 bf16, 44 -> 37 us.
__device__ __forceinline__ void normal_parts2(unsigned long long z, unsigned long long* cdf, unsigned long long* e) {
  using namespace attn_util;
  auto both = [](float v) { return pack2(__float_as_uint(v), __float_as_uint(v)); };
  float z0, z1, x0, x1;
  unpack2(z, z0, z1);
  unpack2(mul2(mul2(both(-0.5f * 1.4426950408889634f), z), z), x0, x1);
  *e = pack2(__float_as_uint(ex2(x0)), __float_as_uint(ex2(x1)));
  unpack2(fma2(both(0.3275911f * 0.70710678118654752f), pack2(__float_as_uint(fabsf(z0)), __float_as_uint(fabsf(z1))), both(1.f)), x0, x1);
  const unsigned long long t = pack2(__float_as_uint(rcp(x0)), __float_as_uint(rcp(x1)));
  unsigned long long poly = fma2(both(1.061405429f), t, both(-1.453152027f));
  poly = fma2(poly, t, both(1.421413741f));
  poly = fma2(poly, t, both(-0.284496736f));
  poly = fma2(poly, t, both(0.254829592f));
  const unsigned long long q = mul2(mul2(mul2(both(0.5f), poly), t), *e);                 // 1 - Phi(|z|)
  float q0, q1, p0, p1;
  unpack2(q, q0, q1);
  unpack2(fma2(q, both(-1.f), both(1.f)), p0, p1);
  *cdf = pack2(__float_as_uint(z0 >= 0.f ? p0 : q0), __float_as_uint(z1 >= 0.f ? p1 : q1));
}

__device__ __forceinline__ void gelu_grad2(float z0, float z1, float* g0, float* g1) {
  using namespace attn_util;
  const unsigned long long z = pack2(__float_as_uint(z0), __float_as_uint(z1));
  const unsigned long long c = pack2(__float_as_uint(0.3989422804014327f), __float_as_uint(0.3989422804014327f));
  unsigned long long cdf, e;
  normal_parts2(z, &cdf, &e);
  unpack2(fma2(mul2(z, c), e, cdf), *g0, *g1);
}

__device__ __forceinline__ void gelu_value2(float z0, float z1, float* y0, float* y1) {
  using namespace attn_util;
  const unsigned long long z = pack2(__float_as_uint(z0), __float_as_uint(z1));
  unsigned long long cdf, e;
  normal_parts2(z, &cdf, &e);
  unpack2(mul2(z, cdf), *y0, *y1);
}

}  // namespace tmpi
