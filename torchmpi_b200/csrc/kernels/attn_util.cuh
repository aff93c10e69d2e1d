// Small arithmetic helpers shared by the attention kernels and the GELU: reciprocal, exp2 on the special-function unit and on the FMA pipe,
// three-input maximum, and the packed two-lane fp32 operations of sm_100.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace attn_util {

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two fp32 values as packed bf16
__device__ __forceinline__ uint32_t pack_bf16(uint32_t lo, uint32_t hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(lo), __uint_as_float(hi));
  return *reinterpret_cast<uint32_t*>(&h);
}

// maxima that are NaN when an operand is
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// two fp32 lanes per instruction
__device__ __forceinline__ unsigned long long pack2(uint32_t lo, uint32_t hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  const unsigned long long m1 = pack2(0xbf800000u, 0xbf800000u);
  return fma2(b, m1, a);                                   // a - b, rounded once
}

// 2^a, 2^b for a, b <= 0 on the FMA pipe (the special-function unit, 4 lanes per scheduler, is the bottleneck of the softmax:
// a share of the exponentials goes here instead): round to an integer n with the 1.5 * 2^23 trick, a cubic for
// 2^(a - n) on [-0.5, 0.5] (relative error 7.5e-5, far below the bf16 rounding of P), and times 2^n.  Like ex2 it flushes
// subnormals: the last product does, so that an argument of -inf (a masked score, clamped to -126) gives exactly 0.
__device__ __forceinline__ unsigned long long ex2_fma2(float a, float b) {
  auto both = [](float v) { return pack2(__float_as_uint(v), __float_as_uint(v)); };
  const unsigned long long x = pack2(__float_as_uint(fmaxf(a, -126.f)), __float_as_uint(fmaxf(b, -126.f)));
  const unsigned long long t = add2(x, both(12582912.f)), f = sub2(x, add2(t, both(-12582912.f)));
  unsigned long long c = fma2(both(0.05517157167196274f), f, both(0.2426111102104187f));
  c = fma2(c, f, both(0.6932610273361206f));
  c = fma2(c, f, both(0.9999280571937561f));
  float t0, t1;
  unpack2(t, t0, t1);
  unsigned long long r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;"
      : "=l"(r) : "l"(c), "l"(pack2((__float_as_uint(t0) << 23) + 0x3f800000u, (__float_as_uint(t1) << 23) + 0x3f800000u)));
  return r;
}

}  // namespace attn_util
