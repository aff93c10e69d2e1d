// Layer normalisation over the last dimension, forward and backward, for [rows, C] activations.
//
// One warp per row: a lane owns C / 32 elements (packs of 16 bytes, strided by the warp so that the
// warp's loads are contiguous), the row statistics are two warp reductions, and the row is read once.
// Backward computes dx and, in the same pass, the lane's share of dgamma and dbeta in registers over
// all the rows its warp visits; the block's warps are summed through shared memory into one partial
// per block and a second kernel adds the partials in block order (deterministic).  A framework
// graph runs this as three kernels with three reads of dy and x (dx, then the two parameter
// reductions).  The reference has no normalisation layer of its own (it trains Torch7 modules).
#include <cuda.h>
#include "pdl.cuh"
#include "sm100_ptx.cuh"
#include "vec.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"
#include <algorithm>

namespace tmpi {

// Set where a backward gave up on a bounded wait.  On the device: nothing has to be allocated on a first call, which may be
// inside a graph capture.
static __device__ int g_ln_status;

constexpr int kLnThreads = 256, kLnWarps = kLnThreads / 32;
constexpr int kLnMaxGrid = 296;           // forward: two blocks per SM; backward (about 200 registers): half of it, one per SM

// NP = packs per lane (C = 32 * NP * V)
template <typename T, int V, int NP>
__global__ void __launch_bounds__(kLnThreads) ln_fwd_kernel(const T* __restrict__ x, const T* __restrict__ gamma,
                                                            const T* __restrict__ beta, T* __restrict__ y,
                                                            float* __restrict__ mean, float* __restrict__ rstd, int rows, float eps) {
  constexpr int C = 32 * NP * V;
  wait_previous(x, gamma, beta);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float g[NP][V], b[NP][V];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    Pack<T, V> gv = ld_pack<T, V>(gamma + (p * 32 + lane) * V), bv = ld_pack<T, V>(beta + (p * 32 + lane) * V);
#pragma unroll
    for (int k = 0; k < V; ++k) { g[p][k] = (float)to_acc<T>(gv.v[k]); b[p][k] = (float)to_acc<T>(bv.v[k]); }
  }
  for (int r = blockIdx.x * kLnWarps + warp; r < rows; r += gridDim.x * kLnWarps) {
    const T* xr = x + (size_t)r * C;
    Pack<T, V> xv[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) xv[p] = ld_pack<T, V>(xr + (p * 32 + lane) * V);
    float s = 0.f;
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int k = 0; k < V; ++k) s += (float)to_acc<T>(xv[p].v[k]);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(~0u, s, o);
    const float mu = s * (1.f / C);
    float q = 0.f;
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int k = 0; k < V; ++k) { const float d = (float)to_acc<T>(xv[p].v[k]) - mu; q += d * d; }
    for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(~0u, q, o);
    const float rs = rsqrtf(q * (1.f / C) + eps);
    if (lane == 0) { mean[r] = mu; rstd[r] = rs; }
    T* yr = y + (size_t)r * C;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      Pack<T, V> o;
#pragma unroll
      for (int k = 0; k < V; ++k)
        o.v[k] = from_acc<T>((typename AccOf<T>::type)(((float)to_acc<T>(xv[p].v[k]) - mu) * rs * g[p][k] + b[p][k]));
      st_pack<T, V>(yr + (p * 32 + lane) * V, o);
    }
  }
}

// Backward: the rows of a warp come through a ring of its own in shared memory, one bulk copy per row and tensor, so that up to
// four rows (16 KB at 1024 bf16 columns) per warp are in flight whatever the registers hold; the sums, 64 per lane there,
// leave no room for a second row in registers, and one row at a time left the memory idle while it was computed.  Measured,
// 8192 x 1024 bf16, back to back: 19.7 -> 11.4 us (50 MB: 7.7 at the copy rate); 14.3 with nothing in L2, 32768 rows 41.7 (31).
// Rows of a warp's ring, 192 KB at most (216 with a third tensor); of the widest rows three took 61.9 us where two take 56.9 (8192 x
// 2048 bf16).  ADD: a third tensor is added to dx, the gradient that reaches x beside the layer norm (of a residual block's
// identity), which an elementwise pass would read and write once more.
__host__ __device__ constexpr int ln_ring(int np, bool add) { return add ? (np <= 4 ? 4 : np <= 6 ? 3 : 2) : np <= 6 ? 4 : 2; }
// One block per SM, by a floor of shared memory and for the register allocation.  The grid is one block per SM, but under a launch
// that overlaps the one before it blocks start as SMs become free, and where several of these fit into one (rows of 1 KB and
// less: 32 to 64 KB each) the first free SMs got several and others none: 32768 x 256, forward and backward, bf16 47.3 us against
// 30.6 with the floor, fp32 50.9 against 36.5; 8192 x 256 18.6 against 12.6 (16.5 when rows came into registers).
constexpr int kLnOneBlock = 116 << 10;
template <typename T, int NP, bool ADD> constexpr int ln_bwd_smem() {
  const int ring = kLnWarps * ln_ring(NP, ADD) * (ADD ? 3 : 2) * 32 * NP * 16, sums = kLnWarps * 2 * 32 * NP * 16 / (int)sizeof(T) * 4;
  const int need = ring > sums ? ring : sums;         // the warps' sums take the ring's place
  return need > kLnOneBlock ? need : kLnOneBlock;
}

// partial[(block * 2 + which) * C + c], which: 0 = dbeta, 1 = dgamma
template <typename T, int V, int NP, bool ADD>
__global__ void __launch_bounds__(kLnThreads, 1) ln_bwd_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ add,
                                                            const T* __restrict__ gamma, const float* __restrict__ mean,
                                                            const float* __restrict__ rstd, T* __restrict__ dx,
                                                            float* __restrict__ partial, int rows) {
  constexpr int C = 32 * NP * V, ROW = C * (int)sizeof(T), RING = ln_ring(NP, ADD), SET = (ADD ? 3 : 2) * ROW;
  extern __shared__ __align__(128) unsigned char ln_smem[];
  __shared__ uint64_t full[kLnWarps][RING];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* ring = ln_smem + warp * RING * SET;
  if (lane == 0) {
    for (int k = 0; k < RING; ++k) sm100::mbar_init(&full[warp][k], 1);
    sm100::fence_barrier_init();
  }
  __syncwarp();
  wait_previous(x, dy, add, gamma, mean, rstd);
  const int first = blockIdx.x * kLnWarps + warp, stride = gridDim.x * kLnWarps;
  auto fetch = [&](long long r, int k) {
    if (r >= rows || lane) return;
    sm100::mbar_expect_tx(&full[warp][k], SET);
    sm100::bulk_load(ring + k * SET, x + (size_t)r * C, ROW, &full[warp][k]);
    sm100::bulk_load(ring + k * SET + ROW, dy + (size_t)r * C, ROW, &full[warp][k]);
    if (ADD) sm100::bulk_load(ring + k * SET + 2 * ROW, add + (size_t)r * C, ROW, &full[warp][k]);
  };
#pragma unroll
  for (int k = 0; k < RING; ++k) fetch((long long)first + (long long)k * stride, k);
  float g[NP][V], db[NP][V], dg[NP][V];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    Pack<T, V> gv = ld_pack<T, V>(gamma + (p * 32 + lane) * V);
#pragma unroll
    for (int k = 0; k < V; ++k) { g[p][k] = (float)to_acc<T>(gv.v[k]); db[p][k] = 0.f; dg[p][k] = 0.f; }
  }
  int k = 0;
  uint32_t phase = 0;
  float mu_next = first < rows ? mean[first] : 0.f, rs_next = first < rows ? rstd[first] : 0.f;
  for (int r = first; r < rows; r += stride) {
    const float mu = mu_next, rs = rs_next;
    if (r + stride < rows) { mu_next = mean[r + stride]; rs_next = rstd[r + stride]; }
    if (!__all_sync(~0u, sm100::mbar_wait(&full[warp][k], phase, 2000000000ull))) {
      if (lane == 0) atomicCAS(&g_ln_status, 0, 4001);
      const unsigned long long t0 = sm100::now_ns();
      while (sm100::now_ns() - t0 < 200000000ull) { __nanosleep(1000); }   // copies in flight land within microseconds
      break;
    }
    const T* row = reinterpret_cast<const T*>(ring + k * SET);
    Pack<T, V> xv[NP], yv[NP], av[ADD ? NP : 1];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      xv[p] = ld_pack<T, V>(row + (p * 32 + lane) * V);
      yv[p] = ld_pack<T, V>(row + C + (p * 32 + lane) * V);
      if (ADD) av[p] = ld_pack<T, V>(row + 2 * C + (p * 32 + lane) * V);
    }
    __syncwarp();                           // the row is in registers
    fetch((long long)r + (long long)RING * stride, k);
    if (++k == RING) { k = 0; phase ^= 1; }
    float s1 = 0.f, s2 = 0.f;               // sum(dy * gamma), sum(dy * gamma * xhat)
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const float d = (float)to_acc<T>(yv[p].v[e]);
        const float xh = ((float)to_acc<T>(xv[p].v[e]) - mu) * rs;
        db[p][e] += d;
        dg[p][e] += d * xh;
        s1 += d * g[p][e];
        s2 += d * g[p][e] * xh;
      }
    for (int o = 16; o; o >>= 1) { s1 += __shfl_xor_sync(~0u, s1, o); s2 += __shfl_xor_sync(~0u, s2, o); }
    s1 *= 1.f / C; s2 *= 1.f / C;
    T* dr = dx + (size_t)r * C;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      Pack<T, V> o;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const float d = (float)to_acc<T>(yv[p].v[e]);
        const float xh = ((float)to_acc<T>(xv[p].v[e]) - mu) * rs;
        float dxv = rs * (d * g[p][e] - s1 - xh * s2);
        if (ADD) dxv += (float)to_acc<T>(av[p].v[e]);
        o.v[e] = from_acc<T>((typename AccOf<T>::type)dxv);
      }
      st_pack<T, V>(dr + (p * 32 + lane) * V, o);
    }
  }
  // the block's eight warps hold the same columns: their sums are added in warp order
  __syncthreads();                          // every row of the ring has been read
  float* mine = reinterpret_cast<float*>(ln_smem) + warp * 2 * C;
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int e = 0; e < V; e += 4) {
      const int c = (p * 32 + lane) * V + e;
      *reinterpret_cast<float4*>(mine + c) = make_float4(db[p][e], db[p][e + 1], db[p][e + 2], db[p][e + 3]);
      *reinterpret_cast<float4*>(mine + C + c) = make_float4(dg[p][e], dg[p][e + 1], dg[p][e + 2], dg[p][e + 3]);
    }
  __syncthreads();
  for (int o = threadIdx.x; o < 2 * C; o += kLnThreads) {
    float t = reinterpret_cast<const float*>(ln_smem)[o];
#pragma unroll
    for (int w = 1; w < kLnWarps; ++w) t += reinterpret_cast<const float*>(ln_smem)[w * 2 * C + o];
    partial[(size_t)blockIdx.x * 2 * C + o] = t;
  }
}

// One block per 32 columns of one of the two sums; 32 warps add a contiguous range of the partial rows each, then warp 0 the 32
// sums in order.  (A thread per column added all rows one after the other: 148 of them took 7.2 us at 1024 columns, now 2.7.)
constexpr int kLnFinGroups = 32;
template <typename T>
__global__ void __launch_bounds__(32 * kLnFinGroups) ln_finalize_kernel(const float* __restrict__ partial, int nblocks, int C,
                                                                        T* __restrict__ dgamma, T* __restrict__ dbeta) {
  wait_previous(partial);
  const int cx = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int o = blockIdx.x * 32 + cx;                       // (which, c); C is a multiple of 32
  const int which = o / C, c = o - which * C;
  const int per = (nblocks + kLnFinGroups - 1) / kLnFinGroups, end = min(nblocks, (grp + 1) * per);
  float t = 0.f;
#pragma unroll 5
  for (int blk = grp * per; blk < end; ++blk) t += partial[((size_t)blk * 2 + which) * C + c];
  __shared__ float s[kLnFinGroups][32];
  s[grp][cx] = t;
  __syncthreads();
  if (grp == 0) {
    float sum = s[0][cx];
#pragma unroll
    for (int g = 1; g < kLnFinGroups; ++g) sum += s[g][cx];
    (which ? dgamma : dbeta)[c] = from_acc<T>((typename AccOf<T>::type)sum);
  }
}

static int ln_grid(int rows) { return std::max(1, std::min((rows + kLnWarps - 1) / kLnWarps, kLnMaxGrid)); }

template <typename T, int NP>
static cudaError_t ln_launch(bool fwd, const void* x, const void* a, const void* add, const void* gamma, const void* beta, void* out, float* mean,
                             float* rstd, float* partial, void* dgamma, void* dbeta, int rows, float eps, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  constexpr int C = 32 * NP * V;
  const int grid = fwd ? ln_grid(rows) : std::min(ln_grid(rows), kLnMaxGrid / 2);
  if (fwd)
    return launch_overlapped(ln_fwd_kernel<T, V, NP>, grid, kLnThreads, 0, s, (const T*)x, (const T*)gamma, (const T*)beta, (T*)out, mean,
                             rstd, rows, eps);
  const auto backward = [&](auto kernel, int smem) -> cudaError_t {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return launch_overlapped(kernel, grid, kLnThreads, smem, s, (const T*)x, (const T*)a, (const T*)add, (const T*)gamma, mean, rstd, (T*)out,
                             partial, rows);
  };
  const cudaError_t e = add ? backward(ln_bwd_kernel<T, V, NP, true>, ln_bwd_smem<T, NP, true>())
                            : backward(ln_bwd_kernel<T, V, NP, false>, ln_bwd_smem<T, NP, false>());
  if (e != cudaSuccess) return e;
  return launch_overlapped(ln_finalize_kernel<T>, 2 * C / 32, 32 * kLnFinGroups, 0, s, partial, grid, C, (T*)dgamma, (T*)dbeta);
}

template <typename T>
static int ln_dispatch(bool fwd, const void* x, const void* a, const void* add, const void* gamma, const void* beta, void* out, float* mean,
                       float* rstd, float* partial, void* dgamma, void* dbeta, int rows, int C, float eps, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  if (!all_aligned16({x, a, add, gamma, beta, out}))
    return fail(TMPI_ERR_INVALID, "layernorm: tensors must be 16-byte aligned");
  if (rows < 1 || C % (32 * V)) return fail(TMPI_ERR_UNSUPPORTED, "layernorm: C=%d must be a multiple of %d", C, 32 * V);
  cudaError_t e;
  switch (C / (32 * V)) {
    case 1: e = ln_launch<T, 1>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    case 2: e = ln_launch<T, 2>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    case 3: e = ln_launch<T, 3>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    case 4: e = ln_launch<T, 4>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    case 5: e = ln_launch<T, 5>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    case 6: e = ln_launch<T, 6>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    case 8: e = ln_launch<T, 8>(fwd, x, a, add, gamma, beta, out, mean, rstd, partial, dgamma, dbeta, rows, eps, s); break;
    default: return fail(TMPI_ERR_UNSUPPORTED, "layernorm: C=%d is not covered (%d elements per lane)", C, C / 32);
  }
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "layernorm launch: %s", cudaGetErrorString(e));
}

}  // namespace tmpi

using namespace tmpi;

extern "C" {

// 1 if tmpi_layernorm_* cover this width and type
int tmpi_layernorm_supported(int channels, int dtype) {
  const int V = dtype == TMPI_F32 ? 4 : 8;
  if (dtype != TMPI_F32 && dtype != TMPI_BF16 && dtype != TMPI_F16) return 0;
  if (channels % (32 * V)) return 0;
  const int np = channels / (32 * V);
  return np >= 1 && np <= 8 && np != 7;
}

size_t tmpi_layernorm_scratch_bytes(int channels) { return (size_t)kLnMaxGrid * 2 * channels * sizeof(float); }

// y = (x - mean) * rstd * gamma + beta per row; mean / rstd ([rows], fp32) are kept for backward.
// gamma, beta, x, y share the dtype.
int tmpi_layernorm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows,
                       int channels, float eps, int dtype, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return ln_dispatch<__nv_bfloat16>(true, x, nullptr, nullptr, gamma, beta, y, mean, rstd, nullptr, nullptr, nullptr, rows, channels, eps, s);
    case TMPI_F16: return ln_dispatch<__half>(true, x, nullptr, nullptr, gamma, beta, y, mean, rstd, nullptr, nullptr, nullptr, rows, channels, eps, s);
    case TMPI_F32: return ln_dispatch<float>(true, x, nullptr, nullptr, gamma, beta, y, mean, rstd, nullptr, nullptr, nullptr, rows, channels, eps, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "layernorm: dtype %d", dtype);
}

// dx, dgamma, dbeta from dy in one pass over (x, dy); scratch: tmpi_layernorm_scratch_bytes(channels).
int tmpi_layernorm_bwd(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx,
                       void* dgamma, void* dbeta, int rows, int channels, int dtype, void* scratch, void* stream) {
  return tmpi_layernorm_bwd_add(x, dy, nullptr, gamma, mean, rstd, dx, dgamma, dbeta, rows, channels, dtype, scratch, stream);
}

// The same with `add`, of x's shape and type, added to dx (null: nothing).
int tmpi_layernorm_bwd_add(const void* x, const void* dy, const void* add, const void* gamma, const float* mean, const float* rstd, void* dx,
                           void* dgamma, void* dbeta, int rows, int channels, int dtype, void* scratch, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  float* m = const_cast<float*>(mean);
  float* r = const_cast<float*>(rstd);
  switch (dtype) {
    case TMPI_BF16: return ln_dispatch<__nv_bfloat16>(false, x, dy, add, gamma, nullptr, dx, m, r, (float*)scratch, dgamma, dbeta, rows, channels, 0.f, s);
    case TMPI_F16: return ln_dispatch<__half>(false, x, dy, add, gamma, nullptr, dx, m, r, (float*)scratch, dgamma, dbeta, rows, channels, 0.f, s);
    case TMPI_F32: return ln_dispatch<float>(false, x, dy, add, gamma, nullptr, dx, m, r, (float*)scratch, dgamma, dbeta, rows, channels, 0.f, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "layernorm: dtype %d", dtype);
}

// Non-zero after a layer-norm backward on the current device gave up on a bounded wait (rows of its dx are missing); clears it.
// Waits for the device's work on the default stream.
int tmpi_layernorm_status(void) {
  int v = 0;
  const int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_ln_status, sizeof(v)) != cudaSuccess) { cudaGetLastError(); return 0; }
  if (v) cudaMemcpyToSymbol(g_ln_status, &zero, sizeof(zero));
  return v;
}

}  // extern "C"
