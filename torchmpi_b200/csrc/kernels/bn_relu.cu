// Fused batch-norm (+ residual add) (+ ReLU), forward and backward, for channels-last activations.
//
// The activation is a [rows, C] matrix (rows = N*H*W, C contiguous).  Training forward:
//   stats    : per-channel sum and sum of squares (one read of x)
//   finalize : mean, 1/std, running statistics (32 x 32 threads per 32 channels)
//   apply    : y = relu((x - mean) * invstd * gamma + beta + residual)   (read x [, residual], write y)
// Backward, with dz = dy * (y > 0):
//   reduce   : dbeta = sum dz, dgamma = sum dz * xhat
//   finalize : (same shape)
//   apply    : dx = gamma * invstd * (dz - dbeta/M - xhat * dgamma/M); dresidual = dz
// A framework graph runs batch-norm, add and ReLU as separate kernels with their own reads and
// writes of the activation; the reference has no such ops at all (its only kernel is `out += in`,
// lib/detail/reduce_kernel.cu).  Every thread owns a fixed group of V channels, so partial sums
// stay in registers; block partials go to scratch and are reduced in block order (deterministic).
// A ReLU layer without a residual does not read y in backward: y > 0 exactly when the affine
// transform of x is positive, and x is read anyway.
#include "vec.cuh"
#include "pool_rows.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"
#include <algorithm>
#include <type_traits>

namespace tmpi {

constexpr int kBnThreads = 256;
constexpr int kBnMaxGrid = 592;     // 148 SMs x 4 resident CTAs

// Blocks of a streaming pass: `most`, or fewer where there are not U vectors for every thread of them; but a block per SM where
// there is one vector each, so that the smallest tensors are not left to a few SMs.
static int bn_grid(size_t nvec, int most, int U) {
  const size_t one = (nvec + kBnThreads - 1) / kBnThreads;
  return (int)std::max<size_t>(1, std::min<size_t>(std::max((one + U - 1) / U, std::min<size_t>(one, 148)), most));
}

// A pack of NW 32-bit words (8 or 16 bytes), elements taken out and put in by shifts and pair conversions (element-wise
// structs cost a register per 16-bit element here and spilled).
template <int NW> struct BpWords { uint32_t w[NW]; };
template <int NW> __device__ __forceinline__ BpWords<NW> bp_ld(const void* p) {
  if constexpr (NW == 4) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    return BpWords<NW>{{u.x, u.y, u.z, u.w}};
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return BpWords<NW>{{u.x, u.y}};
  }
}
template <int NW> __device__ __forceinline__ void bp_st(void* p, const BpWords<NW>& b) {
  if constexpr (NW == 4) *reinterpret_cast<uint4*>(p) = make_uint4(b.w[0], b.w[1], b.w[2], b.w[3]);
  else *reinterpret_cast<uint2*>(p) = make_uint2(b.w[0], b.w[1]);
}
template <typename T, int NW> __device__ __forceinline__ float bp_get(const BpWords<NW>& b, int c) {
  if constexpr (sizeof(T) == 4) return __uint_as_float(b.w[c]);
  else if constexpr (std::is_same<T, __nv_bfloat16>::value) return __uint_as_float((c & 1) ? b.w[c >> 1] & 0xffff0000u : b.w[c >> 1] << 16);
  else return __half2float(__ushort_as_half((unsigned short)((c & 1) ? b.w[c >> 1] >> 16 : b.w[c >> 1])));
}
// from V floats
template <typename T, int V> __device__ __forceinline__ BpWords<V * sizeof(T) / 4> bp_put(const float (&f)[V]) {
  BpWords<V * sizeof(T) / 4> b;
#pragma unroll
  for (int k = 0; k < (int)(V * sizeof(T) / 4); ++k) {
    if constexpr (sizeof(T) == 4) b.w[k] = __float_as_uint(f[k]);
    else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
      b.w[k] = *reinterpret_cast<uint32_t*>(&h);
    } else {
      __half2 h = __floats2half2_rn(f[2 * k], f[2 * k + 1]);
      b.w[k] = *reinterpret_cast<uint32_t*>(&h);
    }
  }
  return b;
}

// The passes stream each tensor once and are bound by memory, so what counts is bytes in flight: each thread issues the loads
// of U vectors before it uses the first, without branches between them (mask source, residual and its gradient are template
// parameters; the loads are volatile to stay in front).  Fewer resident blocks with more registers hold more bytes in flight
// than eight or four small ones.
// Measured, in us, one small vector at a time as it was first, and now: bf16, 256 x 28 x 28 x 512, sums under mask bits 92, 73 (411
// MB: 63 at the copy rate), forward apply with a residual 109, 94 (96), backward apply with the residual's gradient 130, 128;
// 256 x 28 x 28 x 128, sums 30, 23, forward apply 16.5, 14.7, backward apply 28.7, 22.1; fp32, 64 x 56 x 56 x 64, forward apply 12.6,
// 12.1, backward apply 20.5, 19.1.
//
// PAST_L1: loads that allocate nothing in L1.  They are the faster ones where a pass is the first to read what a kernel before it
// has written (the forward apply behind a convolution: inference through a bottleneck of 32 x 56 x 56, 113 us with them and 120
// without, 96 x 28 x 28 220 and 231; the statistics of the stem's 411 MB: 702 and 715 for the stem;
// its backward sums over the kept inputs 757 and 760), and the slower ones where it
// reads again what another pass of the layer has just read (forward apply after the statistics 107 and 94, 20.0 and 14.7, 17.5
// and 12.1 for the sizes above; backward apply after the sums 135 and 128, 27.1 and 22.1, 25.4 and 19.1).
template <bool PAST_L1, typename T>
__device__ __forceinline__ BpWords<4> bn_ld(const T* p) {
  BpWords<4> u;
  if constexpr (PAST_L1)
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(u.w[0]), "=r"(u.w[1]), "=r"(u.w[2]), "=r"(u.w[3]) : "l"(p));
  else
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(u.w[0]), "=r"(u.w[1]), "=r"(u.w[2]), "=r"(u.w[3]) : "l"(p));
  return u;
}
constexpr int kBnReduceU = 4, kBnApplyU = 2;
constexpr int kBnReduceBwdGrid = 296, kBnApplyGrid = 740, kBnApplyBwdGrid = 444;       // resident blocks: 2, 5, 3 per SM

// partial[(block * 2 + which) * C + c]
// Where a backward pass takes the ReLU mask from (a template parameter: a choice at run time puts branches between the loads).
enum { MASK_NONE = 0, MASK_X = 1 /* recomputed from x, gamma, beta */, MASK_BITS = 2, MASK_Y = 3, MASK_X_ROUNDED = 4 /* MASK_X, of the value rounded to T */ };
__host__ __device__ constexpr bool bn_mask_from_x(int mask) { return mask == MASK_X || mask == MASK_X_ROUNDED; }

template <typename T, int V, bool BWD, int MASK, bool PAST_L1>
__global__ void __launch_bounds__(kBnThreads, BWD ? 2 : 4) bn_reduce_kernel(
    const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ dy,
    const float* __restrict__ mean, const float* __restrict__ invstd,
    const float* __restrict__ gamma, const float* __restrict__ beta, const unsigned char* __restrict__ bits,
    size_t nvec, int C, int reverse, float* __restrict__ partial) {
  const int cvn = C / V;
  const size_t T0 = (size_t)blockIdx.x * kBnThreads + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * kBnThreads;
  // reverse: the walk starts at the end of the tensor (vector nvec-1-T0, then down by the stride), where
  // the lines the producer wrote last are still in L2; the apply pass that follows walks up from the
  // start, which this pass read last.  nvec and the stride are multiples of cvn: the group stays fixed.
  const int cv = reverse ? cvn - 1 - (int)(T0 % cvn) : (int)(T0 % cvn);
  float a[V], b[V], mu[V], sc[V], sh[V];
#pragma unroll
  for (int k = 0; k < V; ++k) { a[k] = 0.f; b[k] = 0.f; }
  if constexpr (BWD) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      mu[k] = mean[cv * V + k];
      if constexpr (bn_mask_from_x(MASK)) { sc[k] = invstd[cv * V + k] * gamma[cv * V + k]; sh[k] = beta[cv * V + k] - mu[k] * sc[k]; }
    }
  }
  // bits (backward, ReLU layers with a residual): one byte per vector written by the forward apply
  // pass, bit k set where the output was positive; replaces the read of y
  auto accumulate = [&](const BpWords<4>& xv, const BpWords<4>& gv, const BpWords<4>& yv, unsigned mb) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float f = bp_get<T>(xv, k);
      if constexpr (!BWD) {
        a[k] += f;
        b[k] += f * f;
      } else {
        float g = bp_get<T>(gv, k);
        if (MASK == MASK_X && !(f * sc[k] + sh[k] > 0.f)) g = 0.f;
        if (MASK == MASK_X_ROUNDED && !((float)to_acc<T>(from_acc<T>((typename AccOf<T>::type)(f * sc[k] + sh[k]))) > 0.f)) g = 0.f;
        if (MASK == MASK_BITS && !((mb >> k) & 1u)) g = 0.f;
        if (MASK == MASK_Y && !(bp_get<T>(yv, k) > 0.f)) g = 0.f;
        a[k] += g;
        b[k] += g * (f - mu[k]);             // times 1 / std at the end
      }
    }
  };
  auto pass = [&](size_t v, auto count) {
    constexpr int U = decltype(count)::value;
    BpWords<4> xv[U], gv[U], yv[U];
    unsigned mb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t at = reverse ? nvec - 1 - (v + u * stride) : v + u * stride;
      xv[u] = bn_ld<PAST_L1>(x + at * V);
      mb[u] = 0;
      if constexpr (BWD) {
        gv[u] = bn_ld<PAST_L1>(dy + at * V);
        if constexpr (MASK == MASK_BITS) mb[u] = bits[at];
        if constexpr (MASK == MASK_Y) yv[u] = bn_ld<PAST_L1>(y + at * V);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) accumulate(xv[u], gv[u], yv[u], mb[u]);
  };
  size_t v = T0;
  for (; v + (kBnReduceU - 1) * stride < nvec; v += kBnReduceU * stride) pass(v, std::integral_constant<int, kBnReduceU>());
  for (; v < nvec; v += stride) pass(v, std::integral_constant<int, 1>());
  if constexpr (BWD) {
#pragma unroll
    for (int k = 0; k < V; ++k) b[k] *= invstd[cv * V + k];
  }
  __shared__ float s[kBnThreads][2 * V + 1];
#pragma unroll
  for (int k = 0; k < V; ++k) { s[threadIdx.x][k] = a[k]; s[threadIdx.x][V + k] = b[k]; }
  __syncthreads();
  // thread t < cvn * 2V sums one (channel, which) pair over the threads that share its channel group
  for (int o = threadIdx.x; o < cvn * 2 * V; o += kBnThreads) {
    const int c = o / (2 * V), k = o % (2 * V);   // c: channel group, k: slot
    float t = 0.f;
    for (int g = reverse ? cvn - 1 - c : c; g < kBnThreads; g += cvn) t += s[g][k];   // the threads whose group is c
    const int which = k / V, ch = c * V + (k % V);
    partial[((size_t)blockIdx.x * 2 + which) * C + ch] = t;
  }
}

// Sums the per-block partials of 32 channels with a 32 x 32 thread block: thread (cx, ry) adds the
// blocks ry, ry + 32, ... of channel cx (coalesced over cx), then row 0 adds the 32 slices in order.
// All of a thread's loads are issued before the first add (the trip count is bounded by the largest
// grid): a loop of dependent load-add pairs cost one L2 latency per partial, which made this tiny
// kernel as slow as a bandwidth-bound pass.
// PER loads of each sum for a thread, for up to 32 PER rows: a convolution leaves a row per SM and small tensors fewer, and loads that are
// predicated off still pass through.  The order of the sums is the same.  Forward and backward with 19 throughout and now, us: a
// residual block of 256 x 512 x 28 x 28 988, 971; 16 x 2048 x 7 x 7 186.8, 178.5; the stem of 8 images of 128 x 128 55.5, 51.6.
template <int PER>
__device__ __forceinline__ bool bn_partial_sums_of(const float* __restrict__ partial, int nblocks, int C, float* s1, float* s2) {
  __shared__ float sh1[32][33], sh2[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float va[PER], vb[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int blk = threadIdx.y + 32 * j;
    const bool ok = c < C && blk < nblocks;
    va[j] = ok ? partial[((size_t)blk * 2) * C + c] : 0.f;
    vb[j] = ok ? partial[((size_t)blk * 2 + 1) * C + c] : 0.f;
  }
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int j = 0; j < PER; ++j) { a += va[j]; b += vb[j]; }
  sh1[threadIdx.y][threadIdx.x] = a;
  sh2[threadIdx.y][threadIdx.x] = b;
  __syncthreads();
  if (threadIdx.y != 0 || c >= C) return false;
  a = 0.f; b = 0.f;
#pragma unroll
  for (int r = 0; r < 32; ++r) { a += sh1[r][threadIdx.x]; b += sh2[r][threadIdx.x]; }
  *s1 = a; *s2 = b;
  return true;
}

__device__ __forceinline__ bool bn_partial_sums(const float* __restrict__ partial, int nblocks, int C, float* s1, float* s2) {
  if (nblocks <= 32 * 2) return bn_partial_sums_of<2>(partial, nblocks, C, s1, s2);
  if (nblocks <= 32 * 5) return bn_partial_sums_of<5>(partial, nblocks, C, s1, s2);
  if (nblocks <= 32 * 10) return bn_partial_sums_of<10>(partial, nblocks, C, s1, s2);
  return bn_partial_sums_of<(kBnMaxGrid + 31) / 32>(partial, nblocks, C, s1, s2);
}

__global__ void __launch_bounds__(1024) bn_finalize_fwd_kernel(
    const float* __restrict__ partial, int nblocks, int C, float inv_m, float m_corr, float eps, float momentum,
    float* __restrict__ mean, float* __restrict__ invstd, float* __restrict__ rmean, float* __restrict__ rvar) {
  float s1, s2;
  if (!bn_partial_sums(partial, nblocks, C, &s1, &s2)) return;
  const int c = blockIdx.x * 32 + threadIdx.x;
  const float mu = s1 * inv_m;
  float var = s2 * inv_m - mu * mu;
  if (var < 0.f) var = 0.f;
  mean[c] = mu;
  invstd[c] = rsqrtf(var + eps);
  if (rmean) rmean[c] = (1.f - momentum) * rmean[c] + momentum * mu;
  if (rvar) rvar[c] = (1.f - momentum) * rvar[c] + momentum * var * m_corr;   // unbiased, like torch
}

// acc_gamma / acc_beta (nullable): the parameters' gradient buffers, to which the sums are added as well (the
// caller then needs no separate accumulation kernel)
__global__ void __launch_bounds__(1024) bn_finalize_bwd_kernel(const float* __restrict__ partial, int nblocks, int C,
                                                               float* __restrict__ dgamma, float* __restrict__ dbeta,
                                                               float* __restrict__ acc_gamma = nullptr,
                                                               float* __restrict__ acc_beta = nullptr) {
  float s1, s2;
  if (!bn_partial_sums(partial, nblocks, C, &s1, &s2)) return;
  const int c = blockIdx.x * 32 + threadIdx.x;
  dbeta[c] = s1;
  dgamma[c] = s2;
  if (acc_beta) acc_beta[c] += s1;
  if (acc_gamma) acc_gamma[c] += s2;
}

// RES: a residual is added.  BITS: also write the ReLU mask byte of every vector (residual layers only).
template <typename T, int V, bool RES, bool BITS, bool PAST_L1>
__global__ void __launch_bounds__(kBnThreads, 5) bn_apply_fwd_kernel(
    const T* __restrict__ x, const T* __restrict__ res, T* __restrict__ y, const float* __restrict__ gamma,
    const float* __restrict__ beta, const float* __restrict__ mean, const float* __restrict__ invstd,
    unsigned char* __restrict__ bits, size_t nvec, int C, int relu) {
  const int cvn = C / V;
  const size_t T0 = (size_t)blockIdx.x * kBnThreads + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * kBnThreads;
  const int cv = (int)(T0 % cvn);
  float sc[V], sh[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int c = cv * V + k;
    sc[k] = invstd[c] * gamma[c];
    sh[k] = beta[c] - mean[c] * sc[k];
  }
  auto pass = [&](size_t v, auto count) {
    constexpr int U = decltype(count)::value;
    BpWords<4> xv[U];
    [[maybe_unused]] BpWords<4> rv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      xv[u] = bn_ld<PAST_L1>(x + (v + u * stride) * V);
      if constexpr (RES) rv[u] = bn_ld<PAST_L1>(res + (v + u * stride) * V);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float out[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        float z = bp_get<T>(xv[u], k) * sc[k] + sh[k];
        if constexpr (RES) z += bp_get<T>(rv[u], k);
        if (relu) z = fmaxf(z, 0.f);
        out[k] = z;
      }
      const BpWords<4> o = bp_put<T, V>(out);
      bp_st(y + (v + u * stride) * V, o);
      if (BITS) {
        unsigned mb = 0;
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (bp_get<T>(o, k) > 0.f) mb |= 1u << k;        // what `y > 0` would read back
        bits[v + u * stride] = (unsigned char)mb;
      }
    }
  };
  size_t v = T0;
  for (; v + (kBnApplyU - 1) * stride < nvec; v += kBnApplyU * stride) pass(v, std::integral_constant<int, kBnApplyU>());
  for (; v < nvec; v += stride) pass(v, std::integral_constant<int, 1>());
}

// DRES: the residual's gradient, the masked dy, is written too.
template <typename T, int V, int MASK, bool DRES>
__global__ void __launch_bounds__(kBnThreads, 3) bn_apply_bwd_kernel(
    const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ dy, T* __restrict__ dx,
    T* __restrict__ dres, const float* __restrict__ gamma, const float* __restrict__ beta, const float* __restrict__ mean,
    const float* __restrict__ invstd, const float* __restrict__ dgamma, const float* __restrict__ dbeta,
    const unsigned char* __restrict__ bits, size_t nvec, int C, float inv_m) {
  const int cvn = C / V;
  const size_t T0 = (size_t)blockIdx.x * kBnThreads + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * kBnThreads;
  const int cv = (int)(T0 % cvn);
  float mu[V], k1[V], k2[V], k3[V], sh[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int c = cv * V + k;
    const float is = invstd[c];
    mu[k] = mean[c];
    k1[k] = gamma[c] * is;               // dx = k1 * (dz - k2 - (x - mean) * k3); also the forward scale
    k2[k] = dbeta[c] * inv_m;
    k3[k] = is * dgamma[c] * inv_m;
    sh[k] = MASK == MASK_X ? beta[c] - mu[k] * k1[k] : 0.f;
  }
  auto pass = [&](size_t v, auto count) {
    constexpr int U = decltype(count)::value;
    BpWords<4> xv[U], gv[U], yv[U];
    unsigned mb[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t at = v + u * stride;
      xv[u] = bn_ld<false>(x + at * V);
      gv[u] = bn_ld<false>(dy + at * V);
      mb[u] = 0;
      if constexpr (MASK == MASK_BITS) mb[u] = bits[at];
      if constexpr (MASK == MASK_Y) yv[u] = bn_ld<false>(y + at * V);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float ox[V], og[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const float f = bp_get<T>(xv[u], k);
        float g = bp_get<T>(gv[u], k);
        if (MASK == MASK_X && !(f * k1[k] + sh[k] > 0.f)) g = 0.f;
        if (MASK == MASK_BITS && !((mb[u] >> k) & 1u)) g = 0.f;
        if (MASK == MASK_Y && !(bp_get<T>(yv[u], k) > 0.f)) g = 0.f;
        ox[k] = k1[k] * (g - k2[k] - (f - mu[k]) * k3[k]);
        og[k] = g;
      }
      bp_st(dx + (v + u * stride) * V, bp_put<T, V>(ox));
      if constexpr (DRES) bp_st(dres + (v + u * stride) * V, bp_put<T, V>(og));
    }
  };
  size_t v = T0;
  for (; v + (kBnApplyU - 1) * stride < nvec; v += kBnApplyU * stride) pass(v, std::integral_constant<int, kBnApplyU>());
  for (; v < nvec; v += stride) pass(v, std::integral_constant<int, 1>());
}

static int bn_check(int64_t rows, int C, int V, std::initializer_list<const void*> tensors) {
  if (!all_aligned16(tensors)) return fail(TMPI_ERR_INVALID, "bn: tensors must be 16-byte aligned");
  if (rows < 1 || C < V || C % V) return fail(TMPI_ERR_INVALID, "bn: C=%d must be a multiple of %d", C, V);
  int cvn = C / V;
  if (kBnThreads % cvn) return fail(TMPI_ERR_UNSUPPORTED, "bn: C/%d = %d must divide %d", V, cvn, kBnThreads);
  return TMPI_OK;
}

template <typename T>
static int bn_fwd_t(const void* x, const void* res, void* y, const float* gamma, const float* beta, float* rmean,
                    float* rvar, float* smean, float* sinv, int64_t rows, int C, float eps, float momentum, int relu,
                    int training, void* bits, void* scratch, cudaStream_t s, int given_rows = 0) {
  constexpr int V = 16 / sizeof(T);
  int st = bn_check(rows, C, V, {x, res, y});
  if (st) return st;
  size_t nvec = (size_t)rows * (C / V);
  int grid = bn_grid(nvec, kBnMaxGrid, kBnReduceU);
  const int reverse = tunable("bn_reverse_stats") != 0;
  if (training) {
    // given_rows > 0: the producer of x (a convolution epilogue) has left that many rows of partial sums in scratch
    if (given_rows > 0) grid = given_rows;
    else
    bn_reduce_kernel<T, V, false, MASK_NONE, false><<<grid, kBnThreads, 0, s>>>((const T*)x, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                                     nullptr, nvec, C, reverse, (float*)scratch);
    float m = (float)rows;
    bn_finalize_fwd_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>((const float*)scratch, grid, C, 1.f / m,
                                                           rows > 1 ? m / (m - 1.f) : 1.f, eps, momentum, smean, sinv,
                                                           rmean, rvar);
  }
  const int apply_grid = bn_grid(nvec, kBnApplyGrid, kBnApplyU);
  auto pick = [&](auto past) {
    constexpr bool P = decltype(past)::value;
    return bits ? (res ? bn_apply_fwd_kernel<T, V, true, true, P> : bn_apply_fwd_kernel<T, V, false, true, P>)
                : (res ? bn_apply_fwd_kernel<T, V, true, false, P> : bn_apply_fwd_kernel<T, V, false, false, P>);
  };
  const bool read_before = training && given_rows <= 0;        // by the statistics pass
  const auto apply = read_before ? pick(std::false_type()) : pick(std::true_type());
  apply<<<apply_grid, kBnThreads, 0, s>>>((const T*)x, (const T*)res, (T*)y, gamma, beta, smean, sinv, (unsigned char*)bits, nvec, C, relu);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "bn forward launch: %s", cudaGetErrorString(e));
}

template <typename T>
static int bn_bwd_t(const void* x, const void* y, const void* dy, void* dx, void* dres, const float* gamma,
                    const float* beta, const float* smean, const float* sinv, float* dgamma, float* dbeta, int64_t rows, int C, int relu,
                    const void* bits, void* scratch, cudaStream_t s, float* acc_gamma = nullptr, float* acc_beta = nullptr) {
  constexpr int V = 16 / sizeof(T);
  int st = bn_check(rows, C, V, {x, y, dy, dx, dres});
  if (st) return st;
  if (relu && !y && !bits && (!beta || dres))
    return fail(TMPI_ERR_INVALID, "bn backward: without y or mask bits the layer needs beta and no residual");
  size_t nvec = (size_t)rows * (C / V);
  const int grid = bn_grid(nvec, kBnReduceBwdGrid, kBnReduceU), apply_grid = bn_grid(nvec, kBnApplyBwdGrid, kBnApplyU);
  const int reverse = tunable("bn_reverse_stats") != 0;
  const unsigned char* mb = (const unsigned char*)bits;
  auto passes = [&](auto mode) {
    constexpr int MASK = decltype(mode)::value;
    bn_reduce_kernel<T, V, true, MASK, false><<<grid, kBnThreads, 0, s>>>((const T*)x, (const T*)y, (const T*)dy, smean, sinv, gamma, beta, mb, nvec,
                                                                   C, reverse, (float*)scratch);
    bn_finalize_bwd_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>((const float*)scratch, grid, C, dgamma, dbeta, acc_gamma, acc_beta);
    const auto apply = dres ? bn_apply_bwd_kernel<T, V, MASK, true> : bn_apply_bwd_kernel<T, V, MASK, false>;
    apply<<<apply_grid, kBnThreads, 0, s>>>((const T*)x, (const T*)y, (const T*)dy, (T*)dx, (T*)dres, gamma, beta, smean, sinv, dgamma,
                                            dbeta, mb, nvec, C, 1.f / (float)rows);
  };
  if (!relu) passes(std::integral_constant<int, MASK_NONE>());
  else if (bits) passes(std::integral_constant<int, MASK_BITS>());
  else if (y) passes(std::integral_constant<int, MASK_Y>());
  else passes(std::integral_constant<int, MASK_X>());
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "bn backward launch: %s", cudaGetErrorString(e));
}

// ------------------------------------------------------------------ batch-norm + ReLU + max-pool
// Batch-norm + ReLU + 3x3 / stride-2 / pad-1 max-pool as one stage (the ResNet stem after its
// convolution), for channels-last activations.  The normalised full-resolution activation is never
// written: forward reads the convolution output once and writes the pooled tensor and a one-byte
// window index; backward rebuilds, per input position, the gradient that the pool routes to it
// (from the pooled gradient and the index, which stay in L2) inside both batch-norm backward passes.  Unfused, the same stage writes and re-reads the full-resolution
// activation once forward and its gradient twice backward.
//
//   z = x * scale[c] + shift[c];  a = max(z, 0);  y[oh, ow] = max over the window of a
//   idx = position of the first maximum in the window (kh * 3 + kw), as in pool.cu; 255 where that maximum is 0
//   dz[ih, iw] = sum over windows (oh, ow) covering (ih, iw) with idx == this position of dy[oh, ow]
//   then the usual batch-norm backward on dz.
static_assert(kBpThreads == kBnThreads, "same partial layout as the kernels above");


// Both directions walk down the image in registers: a thread owns one channel pack (16 bytes) of one pooled column and a
// strip of pooled rows, and carries what neighbouring windows share from one row to the next, so that nothing is staged
// in shared memory and no window is scanned position by position.  These stages were bound by instruction issue (a
// window scan of nine compare-and-select steps per channel, address arithmetic per position), at about a quarter of the
// copy bandwidth; see the instruction counts at each kernel.  A pack of neighbouring channels is one full line of x for
// 64 channels, and the column that two neighbours share is an L1 hit.

struct BpWalk { int strips, rows; long long items; };        // strips per image, pooled rows per strip, threads
// Strips of up to 14 pooled rows (a strip re-reads one input row forward, one pooled row backward), shorter ones where
// the launch would otherwise have fewer than four blocks per SM.
template <int V>
static BpWalk bp_walk(const BpDims& d) {
  BpWalk w;
  const long long per_strip = (long long)d.N * d.OW * (d.C / V);
  const long long want = 148LL * 4 * kBpThreads;
  long long strips = (d.OH + 13) / 14;
  strips = std::max(strips, std::min((long long)(d.OH + 1) / 2, (want + per_strip - 1) / per_strip));
  w.rows = (int)((d.OH + strips - 1) / strips);
  w.strips = (d.OH + w.rows - 1) / w.rows;
  w.items = per_strip * w.strips;
  return w;
}
// item t -> channel group (fastest), pooled column, strip, image
__device__ __forceinline__ void bp_item(long long t, int cvn, const BpDims& d, int strips, int* cv, int* ow, int* strip, int* n) {
  long long r = t / cvn;
  *cv = (int)(t - r * cvn);
  const long long q = r / d.OW;
  *ow = (int)(r - q * d.OW);
  *n = (int)(q / strips);
  *strip = (int)(q - (long long)*n * strips);
}

// A window whose maximum is 0 passes no gradient (the ReLU under it is closed everywhere), so its index names no
// position: backward needs no mask of its own.
constexpr uint32_t kBpNowhere = 255;

// One 32-bit word of rectified values (two of a 16-bit type, or one float): batch-norm and ReLU, maximum, and the elements that
// are equal as a mask.  The values are not negative (no -0 either) and not NaN.
template <typename T> struct BpWord {
  static __device__ __forceinline__ uint32_t rectified(uint32_t x, const float* sc, const float* sh) {
    if constexpr (sizeof(T) == 4) {
      return __float_as_uint(fmaxf(__uint_as_float(x) * sc[0] + sh[0], 0.f));
    } else {
      const BpWords<1> w{{x}};
      const float f[2] = {fmaxf(bp_get<T>(w, 0) * sc[0] + sh[0], 0.f), fmaxf(bp_get<T>(w, 1) * sc[1] + sh[1], 0.f)};
      return bp_put<T, 2>(f).w[0];
    }
  }
  static __device__ __forceinline__ uint32_t larger(uint32_t a, uint32_t b) {
    uint32_t r;
    if constexpr (sizeof(T) == 4) r = __float_as_uint(fmaxf(__uint_as_float(a), __uint_as_float(b)));
    else if constexpr (std::is_same<T, __nv_bfloat16>::value) asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    else asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  static __device__ __forceinline__ uint32_t equal(uint32_t a, uint32_t b) {
    uint32_t r;
    if constexpr (sizeof(T) == 4) r = __uint_as_float(a) == __uint_as_float(b) ? ~0u : 0u;
    // bit patterns below 0x8000: 0x8000 minus their difference's bits keeps its top bit only where there is none
    else asm("prmt.b32 %0, %1, %1, 0xbb99;" : "=r"(r) : "r"(0x80008000u - (a ^ b)));
    return r;
  }
};
__device__ __forceinline__ uint32_t bp_select(uint32_t mask, uint32_t a, uint32_t b) { return (mask & a) | (~mask & b); }

// forward: per pooled row two new input rows of three columns each (the third row is the previous pooled row's last one,
// kept as its maximum).  Values are compared two at a time in their 16-bit type, and the first position that equals the
// maximum is selected afterwards together with its input value (32-bit (value, position) keys took more instructions without
// it).  The next pooled row's loads are issued before this one is computed.
// xmax (nullable) receives the input at the maximum: all that the backward sums need of x, a quarter of its size.
// Bound by memory and instruction issue, 565 MB and 103 MB of xmax at 256 x 112 x 112 x 64 bf16 (102 us at the copy rate).
// Measured: 133 us before, without xmax; about 145 with it.
constexpr int kBpV = 4;                                      // channels of a thread
template <typename T>
__global__ void __launch_bounds__(kBpThreads, sizeof(T) == 2 ? 4 : 2) bn_pool_fwd_kernel(
    const T* __restrict__ x, T* __restrict__ y, unsigned char* __restrict__ idx, T* __restrict__ xmax, const float* __restrict__ gamma,
    const float* __restrict__ beta, const float* __restrict__ mean, const float* __restrict__ invstd, BpDims d, BpWalk walk) {
  constexpr int V = kBpV, NW = V * sizeof(T) / 4, E = 4 / sizeof(T);      // words of a pack, elements of a word
  constexpr uint32_t ONES = E == 2 ? 0x00010001u : 1u;      // one per element of a word
  using Words = BpWords<NW>;
  using Word = BpWord<T>;
  const int cvn = d.C / V;
  const long long t = (long long)blockIdx.x * kBpThreads + threadIdx.x;
  if (t >= walk.items) return;
  int cv, ow, strip, n;
  bp_item(t, cvn, d, walk.strips, &cv, &ow, &strip, &n);
  float sc[V], sh[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int c = cv * V + k;
    sc[k] = invstd[c] * gamma[c];
    sh[k] = beta[c] - mean[c] * sc[k];
  }
  const int oh0 = strip * walk.rows, oh1 = min(oh0 + walk.rows, d.OH);
  const size_t line = (size_t)d.W * d.C;
  // A column outside the image counts as 0, which only a window whose maximum is 0 finds; its input is the middle one's,
  // which then is not positive after batch-norm either.
  const uint32_t left = ow > 0 ? ~0u : 0u, right = 2 * ow + 1 < d.W ? ~0u : 0u;
  const T* pc = x + ((size_t)n * d.H + 2 * oh0) * line + (size_t)(2 * ow) * d.C + cv * V;      // input column 2 ow
  const T *pl = left ? pc - d.C : pc, *pr = right ? pc + d.C : pc;
  struct Row { Words l, c, r; };
  auto load = [&](Row& q) { q.l = bp_ld<NW>(pl); q.c = bp_ld<NW>(pc); q.r = bp_ld<NW>(pr); };
  auto down = [&]() { pl += line; pc += line; pr += line; };
  struct Best { uint32_t max[NW], x[NW], at[NW]; };          // of a row or window; `at`: position in it, one per element
  auto row_best = [&](const Row& q) {
    Best b;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const uint32_t l = Word::rectified(q.l.w[w], sc + w * E, sh + w * E) & left, c = Word::rectified(q.c.w[w], sc + w * E, sh + w * E),
                     r = Word::rectified(q.r.w[w], sc + w * E, sh + w * E) & right;
      b.max[w] = Word::larger(l, Word::larger(c, r));
      const uint32_t is_c = Word::equal(c, b.max[w]), is_l = Word::equal(l, b.max[w]);
      b.at[w] = bp_select(is_c, ONES, 2 * ONES) & ~is_l;
      b.x[w] = bp_select(is_l, q.l.w[w], bp_select(is_c, q.c.w[w], q.r.w[w]));
    }
    return b;
  };
  Best above;                                                // the row above the window's middle row
  Row q0, q1;
  if (oh0 > 0) {
    pl -= line; pc -= line; pr -= line;
    load(q0);
    above = row_best(q0);
    down();
  }
  load(q0);
  down();
  if (2 * oh0 + 1 < d.H) load(q1);
  size_t o = (((size_t)n * d.OH + oh0) * d.OW + ow) * d.C + cv * V;
#pragma unroll 1
  for (int oh = oh0; oh < oh1; ++oh, o += (size_t)d.OW * d.C) {
    const Row r0 = q0, r1 = q1;
    if (oh + 1 < oh1) {
      down();
      load(q0);
      down();
      if (2 * oh + 3 < d.H) load(q1);
    }
    const Best mid = row_best(r0);
    Best last;
    if (2 * oh + 1 < d.H) {
      last = row_best(r1);
    } else {                                                 // rows outside the image, like columns
      last = mid;
#pragma unroll
      for (int w = 0; w < NW; ++w) last.max[w] = 0u;
    }
    if (oh == 0) {
      above = mid;
#pragma unroll
      for (int w = 0; w < NW; ++w) above.max[w] = 0u;
    }
    Words ym, xm;
    uint32_t at[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      ym.w[w] = Word::larger(above.max[w], Word::larger(mid.max[w], last.max[w]));
      const uint32_t is_mid = Word::equal(mid.max[w], ym.w[w]), is_above = Word::equal(above.max[w], ym.w[w]);
      xm.w[w] = bp_select(is_above, above.x[w], bp_select(is_mid, mid.x[w], last.x[w]));
      at[w] = bp_select(is_above, above.at[w], bp_select(is_mid, mid.at[w] + 3 * ONES, last.at[w] + 6 * ONES));
    }
    above = last;
    bp_st(y + o, ym);
    uint32_t packed = E == 2 ? __byte_perm(at[0], at[1], 0x6420)
                             : __byte_perm(__byte_perm(at[0], at[1], 0x0040), __byte_perm(at[NW - 2], at[NW - 1], 0x0040), 0x5410);
#pragma unroll
    for (int k = 0; k < V; ++k) {                            // a window whose maximum is 0 names no position
      const uint32_t bits = E == 2 ? (k & 1 ? ym.w[k / 2 % NW] >> 16 : ym.w[k / 2 % NW] & 0xffffu) : ym.w[k % NW];
      if (bits == 0u) packed |= kBpNowhere << (8 * k);
    }
    *reinterpret_cast<uint32_t*>(idx + o) = packed;
    if (xmax) bp_st(xmax + o, xm);
  }
}

// backward: the four input positions (2k + r, 2j + c) of a pooled position (k, j) are covered by the windows (k, j),
// (k, j + 1), (k + 1, j) and (k + 1, j + 1) only, with one fixed code each: nine compare-and-add steps per channel for
// four positions, and the lower two windows are the next row's upper two.
template <typename T, int V>
struct BpWindow {
  static constexpr int NW = V * sizeof(T) / 4;
  BpWords<NW> g;
  uint32_t ix[V / 4];
  __device__ __forceinline__ void load(const T* dy, const unsigned char* idx, size_t at, bool inside) {
#pragma unroll
    for (int k = 0; k < NW; ++k) g.w[k] = 0u;
#pragma unroll
    for (int k = 0; k < V / 4; ++k) ix[k] = 0xffffffffu;
    if (inside) {
      g = bp_ld<NW>(dy + at);
      if constexpr (V == 8) { const uint2 u = *reinterpret_cast<const uint2*>(idx + at); ix[0] = u.x; ix[V / 4 - 1] = u.y; }
      else ix[0] = *reinterpret_cast<const uint32_t*>(idx + at);
    }
  }
  __device__ __forceinline__ uint32_t index(int c) const { return (ix[c >> 2] >> (8 * (c & 3))) & 0xffu; }
};
// gradient that the pool routes to channel c of the four positions, in row-major order
template <typename T, int V>
__device__ __forceinline__ void bp_route(const BpWindow<T, V> (&w)[2][2], int c, float (&g)[4]) {
  const float g00 = bp_get<T>(w[0][0].g, c), g01 = bp_get<T>(w[0][1].g, c), g10 = bp_get<T>(w[1][0].g, c), g11 = bp_get<T>(w[1][1].g, c);
  const uint32_t i00 = w[0][0].index(c), i01 = w[0][1].index(c), i10 = w[1][0].index(c), i11 = w[1][1].index(c);
  g[0] = i00 == 4 ? g00 : 0.f;
  g[1] = i00 == 5 ? g00 : 0.f;
  if (i01 == 3) g[1] += g01;
  g[2] = i00 == 7 ? g00 : 0.f;
  if (i10 == 1) g[2] += g10;
  g[3] = i00 == 8 ? g00 : 0.f;
  if (i01 == 6) g[3] += g01;
  if (i10 == 2) g[3] += g10;
  if (i11 == 0) g[3] += g11;
}

// Walks the strips of this thread's items; use(xv, at, off, w, inside): the packs of the four positions, the first one's
// element and the others' distances from it, the four windows and which positions exist.  The channel group is the same for every item of a thread (the stride is a
// multiple of the number of groups).
template <typename T, int V, typename Use>
__device__ __forceinline__ void bp_walk_strips(const T* __restrict__ x, const T* __restrict__ dy, const unsigned char* __restrict__ idx,
                                               const BpDims& d, const BpWalk& walk, Use use) {
  const int cvn = d.C / V;
  const size_t line = (size_t)d.W * d.C;
  for (long long t = (long long)blockIdx.x * kBpThreads + threadIdx.x; t < walk.items; t += (long long)gridDim.x * kBpThreads) {
    int cv, ow, strip, n;
    bp_item(t, cvn, d, walk.strips, &cv, &ow, &strip, &n);
    const int k0 = strip * walk.rows, k1 = min(k0 + walk.rows, d.OH);
    const bool right = ow + 1 < d.OW, odd = 2 * ow + 1 < d.W;
    size_t o = (((size_t)n * d.OH + k0) * d.OW + ow) * d.C + cv * V;
    size_t at = ((size_t)n * d.H + 2 * k0) * line + (size_t)(2 * ow) * d.C + cv * V;
    BpWindow<T, V> w[2][2];
    w[0][0].load(dy, idx, o, true);
    w[0][1].load(dy, idx, o + d.C, right);
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      o += (size_t)d.OW * d.C;
      const bool lower = k + 1 < d.OH, low_row = 2 * k + 1 < d.H;
      const bool in[4] = {true, odd, low_row, odd && low_row};
      const int off[4] = {0, d.C, (int)line, (int)line + d.C};
      BpWords<V * sizeof(T) / 4> xv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (in[q]) xv[q] = bp_ld<V * sizeof(T) / 4>(x + at + off[q]);
      w[1][0].load(dy, idx, o, lower);
      w[1][1].load(dy, idx, o + d.C, lower && right);
      use(xv, at, off, w, in);
      w[0][0] = w[1][0];
      w[0][1] = w[1][1];
      at += 2 * line;
    }
  }
}

// backward statistics without the kept inputs: sums of dz and dz * (x - mean) per channel over all positions of x, one partial
// row per block.  256 x 112 x 112 x 64 bf16: 137 us, against 36 over the kept inputs.
template <typename T, int V, int BLOCKS>
__global__ void __launch_bounds__(kBpThreads, BLOCKS) bn_pool_bwd_reduce_kernel(
    const T* __restrict__ x, const T* __restrict__ dy, const unsigned char* __restrict__ idx, const float* __restrict__ mean,
    const float* __restrict__ invstd, BpDims d, BpWalk walk, float* __restrict__ partial) {
  const int cvn = d.C / V, cv = threadIdx.x % cvn;                // kBpThreads is a multiple of cvn
  float a[V], b[V], mu[V];
#pragma unroll
  for (int k = 0; k < V; ++k) { a[k] = 0.f; b[k] = 0.f; mu[k] = mean[cv * V + k]; }
  bp_walk_strips<T, V>(x, dy, idx, d, walk, [&](const BpWords<V * sizeof(T) / 4> (&xv)[4], size_t, const int (&)[4], const BpWindow<T, V> (&w)[2][2], const bool (&in)[4]) {
#pragma unroll
    for (int c = 0; c < V; ++c) {
      float g[4];
      bp_route<T, V>(w, c, g);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (!in[q]) continue;
        a[c] += g[q];
        b[c] += g[q] * (bp_get<T>(xv[q], c) - mu[c]);
      }
    }
  });
  __shared__ float s[kBpThreads][2 * V + 1];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    s[threadIdx.x][k] = a[k];
    s[threadIdx.x][V + k] = b[k] * invstd[cv * V + k];
  }
  __syncthreads();
  for (int o = threadIdx.x; o < cvn * 2 * V; o += kBpThreads) {
    const int c = o / (2 * V), k = o % (2 * V);
    float t = 0.f;
    for (int g = c; g < kBpThreads; g += cvn) t += s[g][k];
    const int which = k / V, ch = c * V + (k % V);
    partial[((size_t)blockIdx.x * 2 + which) * d.C + ch] = t;
  }
}

// backward apply; measured, 256 x 112 x 112 x 64 bf16: 179 us (208 with the gradient that the pool had written, 411 MB, to read).
template <typename T, int V, int BLOCKS>
__global__ void __launch_bounds__(kBpThreads, BLOCKS) bn_pool_bwd_apply_kernel(
    const T* __restrict__ x, const T* __restrict__ dy, const unsigned char* __restrict__ idx, T* __restrict__ dx,
    const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ invstd, const float* __restrict__ dgamma,
    const float* __restrict__ dbeta, BpDims d, BpWalk walk, float inv_m) {
  const int cvn = d.C / V, cv = threadIdx.x % cvn;                // kBpThreads is a multiple of cvn
  // dx = k1 * (dz - dbeta/M - xhat * dgamma/M) with xhat = (x - mean) * invstd, folded to k1 * dz + ca * x + cb
  float k1[V], ca[V], cb[V];
#pragma unroll
  for (int c = 0; c < V; ++c) {
    const int ch = cv * V + c;
    const float mu = mean[ch], is = invstd[ch];
    k1[c] = gamma[ch] * is;
    ca[c] = -k1[c] * dgamma[ch] * inv_m * is;
    cb[c] = -k1[c] * dbeta[ch] * inv_m - ca[c] * mu;
  }
  bp_walk_strips<T, V>(x, dy, idx, d, walk, [&](const BpWords<V * sizeof(T) / 4> (&xv)[4], size_t at, const int (&off)[4], const BpWindow<T, V> (&w)[2][2], const bool (&in)[4]) {
    // two channels at a time: a pair of results is one word of a 16-bit pack
    BpWords<V * sizeof(T) / 4> ox[4];
#pragma unroll
    for (int c = 0; c < V; c += 2) {
      float g[2][4], r[4][2];
      bp_route<T, V>(w, c, g[0]);
      bp_route<T, V>(w, c + 1, g[1]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e) r[q][e] = k1[c + e] * g[e][q] + ca[c + e] * bp_get<T>(xv[q], c + e) + cb[c + e];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if constexpr (sizeof(T) == 4) { ox[q].w[c] = __float_as_uint(r[q][0]); ox[q].w[c + 1] = __float_as_uint(r[q][1]); }
        else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
          __nv_bfloat162 h = __floats2bfloat162_rn(r[q][0], r[q][1]);
          ox[q].w[c / 2] = *reinterpret_cast<uint32_t*>(&h);
        } else {
          __half2 h = __floats2half2_rn(r[q][0], r[q][1]);
          ox[q].w[c / 2] = *reinterpret_cast<uint32_t*>(&h);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (in[q]) bp_st(dx + at + off[q], ox[q]);
  });
}

// What both directions take, checked before anything is launched: the kernels stage nothing, so a row of any length that an
// int can index.
static int bn_pool_check(int64_t rows, const BpDims& d, int V, const void* idx, std::initializer_list<const void*> tensors) {
  int st = bn_check(rows, d.C, V, tensors);
  if (st) return st;
  if ((uintptr_t)idx % V) return fail(TMPI_ERR_INVALID, "bn+pool: the index must be %d-byte aligned", V);
  if ((int64_t)(d.W + 1) * d.C > 0x7fffffffLL) return fail(TMPI_ERR_UNSUPPORTED, "bn+pool: rows of %d x %d are too long", d.W, d.C);
  return TMPI_OK;
}

template <typename T>
static int bn_pool_fwd_t(const void* x, void* y, void* idx, void* xmax, const float* gamma, const float* beta, float* rmean, float* rvar,
                         float* smean, float* sinv, int N, int H, int W, int C, float eps, float momentum, int training,
                         void* scratch, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const int64_t rows = (int64_t)N * H * W;
  BpDims d{N, H, W, C, (H - 1) / 2 + 1, (W - 1) / 2 + 1};
  int st = bn_pool_check(rows, d, V, idx, {x, y, xmax});
  if (st) return st;
  if (training) {
    size_t nvec = (size_t)rows * (C / V);
    const int grid = bn_grid(nvec, kBnMaxGrid, kBnReduceU);
    bn_reduce_kernel<T, V, false, MASK_NONE, true><<<grid, kBnThreads, 0, s>>>((const T*)x, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                                     nullptr, nvec, C, tunable("bn_reverse_stats") != 0, (float*)scratch);
    float m = (float)rows;
    bn_finalize_fwd_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>((const float*)scratch, grid, C, 1.f / m,
                                                           rows > 1 ? m / (m - 1.f) : 1.f, eps, momentum, smean, sinv, rmean, rvar);
  }
  const BpWalk walk = bp_walk<kBpV>(d);
  bn_pool_fwd_kernel<T><<<(unsigned)((walk.items + kBpThreads - 1) / kBpThreads), kBpThreads, 0, s>>>(
      (const T*)x, (T*)y, (unsigned char*)idx, (T*)xmax, gamma, beta, smean, sinv, d, walk);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "bn+pool forward launch: %s", cudaGetErrorString(e));
}

// returns the rows of partial sums: one resident wave of blocks
template <typename T, int V, int BLOCKS>
static int bn_pool_bwd_reduce(const void* x, const void* dy, const void* idx, const float* smean, const float* sinv, const BpDims& d,
                              void* scratch, cudaStream_t s) {
  static_assert(148 * BLOCKS <= kBnMaxGrid, "partial rows in scratch");
  const BpWalk walk = bp_walk<V>(d);
  const int grid = (int)std::min<long long>((walk.items + kBpThreads - 1) / kBpThreads, 148 * BLOCKS);
  bn_pool_bwd_reduce_kernel<T, V, BLOCKS><<<grid, kBpThreads, 0, s>>>((const T*)x, (const T*)dy, (const unsigned char*)idx, smean, sinv, d,
                                                                      walk, (float*)scratch);
  return grid;
}

template <typename T, int V, int BLOCKS>
static void bn_pool_bwd_apply(const void* x, const void* dy, const void* idx, void* dx, const float* gamma, const float* smean,
                              const float* sinv, const float* dgamma, const float* dbeta, const BpDims& d, cudaStream_t s) {
  const BpWalk walk = bp_walk<V>(d);
  bn_pool_bwd_apply_kernel<T, V, BLOCKS><<<(unsigned)((walk.items + kBpThreads - 1) / kBpThreads), kBpThreads, 0, s>>>(
      (const T*)x, (const T*)dy, (const unsigned char*)idx, (T*)dx, gamma, smean, sinv, dgamma, dbeta, d, walk,
      1.f / (float)((int64_t)d.N * d.H * d.W));
}

template <typename T>
static int bn_pool_bwd_t(const void* x, const void* xmax, const void* dy, const void* idx, void* dx, const float* gamma, const float* beta,
                         const float* smean, const float* sinv, float* dgamma, float* dbeta, int N, int H, int W, int C,
                         void* scratch, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const int64_t rows = (int64_t)N * H * W;
  BpDims d{N, H, W, C, (H - 1) / 2 + 1, (W - 1) / 2 + 1};
  int st = bn_pool_check(rows, d, V, idx, {x, xmax, dy, dx});
  if (st) return st;
  const bool fours = sizeof(T) == 2 && kBpThreads % (C / 4) == 0;       // packs of four channels, see below
  int grid;
  if (xmax) {
    // The sums: dz is zero but at the maximum of each open window, so they run over the pooled positions, with the input that
    // the forward kept for each and the ReLU mask that it implies.  256 x 112 x 112 x 64 bf16: 36 us (206 MB; 136 over
    // all positions of x, 411 MB, with the gradient routed to each).
    const size_t nvec = (size_t)N * d.OH * d.OW * (C / V);
    grid = bn_grid(nvec, kBnReduceBwdGrid, kBnReduceU);
    bn_reduce_kernel<T, V, true, MASK_X_ROUNDED, true><<<grid, kBnThreads, 0, s>>>((const T*)xmax, nullptr, (const T*)dy, smean, sinv, gamma, beta,
                                                                             nullptr, nvec, C, tunable("bn_reverse_stats") != 0, (float*)scratch);
  } else if (fours) {
    grid = bn_pool_bwd_reduce<T, sizeof(T) == 2 ? 4 : V, sizeof(T) == 2 ? 3 : 2>(x, dy, idx, smean, sinv, d, scratch, s);
  } else {
    grid = bn_pool_bwd_reduce<T, V, 2>(x, dy, idx, smean, sinv, d, scratch, s);
  }
  bn_finalize_bwd_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>((const float*)scratch, grid, C, dgamma, dbeta);
  // 16-bit types: packs of four channels where their groups divide the block (up to 1024 channels).  They halve the
  // per-channel state, so that three blocks fit on an SM instead of two (256 x 112 x 112 x 64: 254 -> 179 us).
  if constexpr (sizeof(T) == 2) {
    if (fours) bn_pool_bwd_apply<T, 4, 3>(x, dy, idx, dx, gamma, smean, sinv, dgamma, dbeta, d, s);
    else bn_pool_bwd_apply<T, V, 2>(x, dy, idx, dx, gamma, smean, sinv, dgamma, dbeta, d, s);
  } else {
    bn_pool_bwd_apply<T, V, 2>(x, dy, idx, dx, gamma, smean, sinv, dgamma, dbeta, d, s);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "bn+pool backward launch: %s", cudaGetErrorString(e));
}

}  // namespace tmpi

using namespace tmpi;

extern "C" {

size_t tmpi_bn_scratch_bytes(int channels) { return (size_t)kBnMaxGrid * 2 * channels * sizeof(float); }

// training != 0: batch statistics are computed, saved in save_mean / save_invstd and folded into the
// running statistics.  training == 0: save_mean / save_invstd are inputs (mean and 1/std to apply).
// mask_bits (nullable): one byte per 16-byte vector of y, bit k set where element k is positive; the
// backward of a ReLU layer reads it in place of y.
int tmpi_bn_relu_fwd(const void* x, const void* residual, void* y, const float* gamma, const float* beta,
                     float* running_mean, float* running_var, float* save_mean, float* save_invstd, int64_t rows,
                     int channels, float eps, float momentum, int relu, int training, int dtype, void* mask_bits,
                     void* scratch, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return bn_fwd_t<__nv_bfloat16>(x, residual, y, gamma, beta, running_mean, running_var, save_mean,
                                                   save_invstd, rows, channels, eps, momentum, relu, training, mask_bits, scratch, s);
    case TMPI_F16: return bn_fwd_t<__half>(x, residual, y, gamma, beta, running_mean, running_var, save_mean, save_invstd,
                                           rows, channels, eps, momentum, relu, training, mask_bits, scratch, s);
    case TMPI_F32: return bn_fwd_t<float>(x, residual, y, gamma, beta, running_mean, running_var, save_mean, save_invstd,
                                          rows, channels, eps, momentum, relu, training, mask_bits, scratch, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "bn: dtype %d", dtype);
}

// Training forward whose statistics pass has been done already: `partials` holds `partial_rows` (<= 592) rows of
// per-channel partial sums and sums of squares of x, [row][2][channels] floats, as tmpi_conv_fwd writes them.
int tmpi_bn_relu_fwd_partials(const void* x, const void* residual, void* y, const float* gamma, const float* beta,
                              float* running_mean, float* running_var, float* save_mean, float* save_invstd, int64_t rows,
                              int channels, float eps, float momentum, int relu, int dtype, void* mask_bits,
                              void* partials, int partial_rows, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (partial_rows < 1 || partial_rows > kBnMaxGrid) return fail(TMPI_ERR_INVALID, "bn: 1..%d rows of partial sums", kBnMaxGrid);
  if (dtype != TMPI_BF16) return fail(TMPI_ERR_UNSUPPORTED, "bn from partial sums: bf16 only");
  return bn_fwd_t<__nv_bfloat16>(x, residual, y, gamma, beta, running_mean, running_var, save_mean, save_invstd, rows, channels,
                                 eps, momentum, relu, 1, mask_bits, partials, s, partial_rows);
}

// The ReLU mask comes from mask_bits when given (see tmpi_bn_relu_fwd), else from y, else - ReLU layers
// without a residual only - it is recomputed from x, gamma and beta.
int tmpi_bn_relu_bwd(const void* x, const void* y, const void* dy, void* dx, void* dresidual, const float* gamma,
                     const float* beta, const float* save_mean, const float* save_invstd, float* dgamma, float* dbeta, int64_t rows,
                     int channels, int relu, int dtype, const void* mask_bits, void* scratch, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return bn_bwd_t<__nv_bfloat16>(x, y, dy, dx, dresidual, gamma, beta, save_mean, save_invstd, dgamma, dbeta,
                                                   rows, channels, relu, mask_bits, scratch, s);
    case TMPI_F16: return bn_bwd_t<__half>(x, y, dy, dx, dresidual, gamma, beta, save_mean, save_invstd, dgamma, dbeta, rows,
                                           channels, relu, mask_bits, scratch, s);
    case TMPI_F32: return bn_bwd_t<float>(x, y, dy, dx, dresidual, gamma, beta, save_mean, save_invstd, dgamma, dbeta, rows,
                                          channels, relu, mask_bits, scratch, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "bn: dtype %d", dtype);
}

// tmpi_bn_relu_bwd that also adds dgamma / dbeta to acc_gamma / acc_beta (the parameters' gradient buffers; nullable).
int tmpi_bn_relu_bwd_acc(const void* x, const void* y, const void* dy, void* dx, void* dresidual, const float* gamma,
                         const float* beta, const float* save_mean, const float* save_invstd, float* dgamma, float* dbeta,
                         int64_t rows, int channels, int relu, int dtype, const void* mask_bits, void* scratch,
                         float* acc_gamma, float* acc_beta, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return bn_bwd_t<__nv_bfloat16>(x, y, dy, dx, dresidual, gamma, beta, save_mean, save_invstd, dgamma, dbeta,
                                                   rows, channels, relu, mask_bits, scratch, s, acc_gamma, acc_beta);
    case TMPI_F16: return bn_bwd_t<__half>(x, y, dy, dx, dresidual, gamma, beta, save_mean, save_invstd, dgamma, dbeta, rows,
                                           channels, relu, mask_bits, scratch, s, acc_gamma, acc_beta);
    case TMPI_F32: return bn_bwd_t<float>(x, y, dy, dx, dresidual, gamma, beta, save_mean, save_invstd, dgamma, dbeta, rows,
                                          channels, relu, mask_bits, scratch, s, acc_gamma, acc_beta);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "bn: dtype %d", dtype);
}

// Batch-norm + ReLU + max-pool (3x3, stride 2, pad 1) in one stage.  x: [N, H, W, C] channels-last;
// y, idx: [N, OH, OW, C] with OH = (H - 1) / 2 + 1.  Other arguments as tmpi_bn_relu_fwd / _bwd.
// xmax (nullable): [N, OH, OW, C], the input at each window's maximum; backward forms its sums from it, or over x without it.
int tmpi_bn_relu_pool_fwd_keep(const void* x, void* y, void* idx, void* xmax, const float* gamma, const float* beta, float* running_mean,
                               float* running_var, float* save_mean, float* save_invstd, int N, int H, int W, int channels,
                          float eps, float momentum, int training, int dtype, void* scratch, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return bn_pool_fwd_t<__nv_bfloat16>(x, y, idx, xmax, gamma, beta, running_mean, running_var, save_mean, save_invstd,
                                                        N, H, W, channels, eps, momentum, training, scratch, s);
    case TMPI_F16: return bn_pool_fwd_t<__half>(x, y, idx, xmax, gamma, beta, running_mean, running_var, save_mean, save_invstd, N, H, W,
                                                channels, eps, momentum, training, scratch, s);
    case TMPI_F32: return bn_pool_fwd_t<float>(x, y, idx, xmax, gamma, beta, running_mean, running_var, save_mean, save_invstd, N, H, W,
                                               channels, eps, momentum, training, scratch, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "bn+pool: dtype %d", dtype);
}

int tmpi_bn_relu_pool_bwd_kept(const void* x, const void* xmax, const void* dy, const void* idx, void* dx, const float* gamma, const float* beta,
                          const float* save_mean, const float* save_invstd, float* dgamma, float* dbeta, int N, int H, int W,
                          int channels, int dtype, void* scratch, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return bn_pool_bwd_t<__nv_bfloat16>(x, xmax, dy, idx, dx, gamma, beta, save_mean, save_invstd, dgamma, dbeta, N, H, W,
                                                        channels, scratch, s);
    case TMPI_F16: return bn_pool_bwd_t<__half>(x, xmax, dy, idx, dx, gamma, beta, save_mean, save_invstd, dgamma, dbeta, N, H, W, channels,
                                                scratch, s);
    case TMPI_F32: return bn_pool_bwd_t<float>(x, xmax, dy, idx, dx, gamma, beta, save_mean, save_invstd, dgamma, dbeta, N, H, W, channels,
                                               scratch, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "bn+pool: dtype %d", dtype);
}

int tmpi_bn_relu_pool_fwd(const void* x, void* y, void* idx, const float* gamma, const float* beta, float* running_mean,
                          float* running_var, float* save_mean, float* save_invstd, int N, int H, int W, int channels,
                          float eps, float momentum, int training, int dtype, void* scratch, void* stream) {
  return tmpi_bn_relu_pool_fwd_keep(x, y, idx, nullptr, gamma, beta, running_mean, running_var, save_mean, save_invstd, N, H, W, channels,
                                    eps, momentum, training, dtype, scratch, stream);
}

int tmpi_bn_relu_pool_bwd(const void* x, const void* dy, const void* idx, void* dx, const float* gamma, const float* beta,
                          const float* save_mean, const float* save_invstd, float* dgamma, float* dbeta, int N, int H, int W,
                          int channels, int dtype, void* scratch, void* stream) {
  return tmpi_bn_relu_pool_bwd_kept(x, nullptr, dy, idx, dx, gamma, beta, save_mean, save_invstd, dgamma, dbeta, N, H, W, channels, dtype,
                                    scratch, stream);
}

}  // extern "C"
