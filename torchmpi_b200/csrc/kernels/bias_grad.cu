// Bias gradient of a linear layer, optionally fused with the GELU backward that precedes it:
//   dz = dy * gelu'(z)   (written; skipped when z == nullptr, then dz = dy)
//   db[c] = sum over rows of dz[r, c]
// One pass over dy (and z): a framework graph runs the GELU backward and the column sum as two
// kernels, the second re-reading dz.  Columns are processed in slabs of 1024 (128 threads x one
// 16-byte pack), two rows at a time per block; every thread keeps its eight column sums in
// registers, blocks write partials and a second kernel adds them in block order (deterministic).
// The GELU forward with the same approximation of the normal distribution lives here too.
#include "gelu.cuh"
#include "pdl.cuh"
#include "vec.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"
#include <algorithm>

namespace tmpi {

constexpr int kBgThreads = 256, kBgCols = 128;      // 128 column groups x 2 rows per block
constexpr int kBgMaxRowBlocks = 4 * 148;            // partial rows the scratch buffer holds
constexpr int kBgFinCols = 32, kBgFinGroups = 32;   // finalize: 32 columns x 32 groups of partial rows per block

// y = gelu(z), one 16-byte pack per thread and step, four steps in flight.
template <typename T, int V>
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const T* __restrict__ z, T* __restrict__ y, size_t npacks) {
  wait_previous(z);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int U = 4;
  for (; i + (U - 1) * stride < npacks; i += U * stride) {
    Pack<T, V> a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] = ld_pack<T, V>(z + (i + u * stride) * V);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      Pack<T, V> o;
#pragma unroll
      for (int k = 0; k < V; k += 2) {
        float y0, y1;
        gelu_value2((float)to_acc<T>(a[u].v[k]), (float)to_acc<T>(a[u].v[k + 1]), &y0, &y1);
        o.v[k] = from_acc<T>((typename AccOf<T>::type)y0); o.v[k + 1] = from_acc<T>((typename AccOf<T>::type)y1);
      }
      st_pack<T, V>(y + (i + u * stride) * V, o);
    }
  }
  for (; i < npacks; i += stride) {
    Pack<T, V> a = ld_pack<T, V>(z + i * V), o;
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      float y0, y1;
      gelu_value2((float)to_acc<T>(a.v[k]), (float)to_acc<T>(a.v[k + 1]), &y0, &y1);
      o.v[k] = from_acc<T>((typename AccOf<T>::type)y0); o.v[k + 1] = from_acc<T>((typename AccOf<T>::type)y1);
    }
    st_pack<T, V>(y + i * V, o);
  }
}

template <typename T>
static int gelu_fwd_t(const void* z, void* y, size_t n, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  if (n % V || ((uintptr_t)z & 15) || ((uintptr_t)y & 15))
    return fail(TMPI_ERR_UNSUPPORTED, "gelu_fwd: n=%zu must be a multiple of %d and the pointers 16-byte aligned", n, V);
  const size_t npacks = n / V;
  if (!npacks) return TMPI_OK;
  const int blocks = (int)std::min<size_t>((npacks + 255) / 256, (size_t)148 * 8);
  cudaError_t e = launch_overlapped(gelu_fwd_kernel<T, V>, blocks, 256, 0, s, (const T*)z, (T*)y, npacks);
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "gelu_fwd launch: %s", cudaGetErrorString(e));
}

// dz = dy * gelu'(z), packs as above.  Bound by memory: 8192 x 4096 bf16 33.1 us, 0.93 of the copy rate, with two packs of each operand in
// flight and four blocks per SM; 50.2 with four packs and the registers that they take.  The pass below, with the column sums,
// takes 42.4.
template <typename T, int V>
__global__ void __launch_bounds__(256, 4) gelu_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ z, T* __restrict__ dz, size_t npacks) {
  wait_previous(dy, z);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int U = 2;
  auto one = [&](const Pack<T, V>& g, const Pack<T, V>& a, size_t at) {
    Pack<T, V> o;
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      float d[2];
      gelu_grad2((float)to_acc<T>(a.v[k]), (float)to_acc<T>(a.v[k + 1]), &d[0], &d[1]);
#pragma unroll
      for (int e = 0; e < 2; ++e) o.v[k + e] = from_acc<T>((typename AccOf<T>::type)((float)to_acc<T>(g.v[k + e]) * d[e]));
    }
    st_pack<T, V>(dz + at * V, o);
  };
  for (; i + (U - 1) * stride < npacks; i += U * stride) {
    Pack<T, V> g[U], a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) { g[u] = ld_pack<T, V>(dy + (i + u * stride) * V); a[u] = ld_pack<T, V>(z + (i + u * stride) * V); }
#pragma unroll
    for (int u = 0; u < U; ++u) one(g[u], a[u], i + u * stride);
  }
  for (; i < npacks; i += stride) one(ld_pack<T, V>(dy + i * V), ld_pack<T, V>(z + i * V), i);
}

template <typename T>
static int gelu_bwd_t(const void* dy, const void* z, void* dz, size_t n, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  if (n % V || (((uintptr_t)dy | (uintptr_t)z | (uintptr_t)dz) & 15))
    return fail(TMPI_ERR_UNSUPPORTED, "gelu_bwd: n=%zu must be a multiple of %d and the pointers 16-byte aligned", n, V);
  const size_t npacks = n / V;
  if (!npacks) return TMPI_OK;
  const int blocks = (int)std::min<size_t>((npacks + 255) / 256, (size_t)148 * 4);
  cudaError_t e = launch_overlapped(gelu_bwd_kernel<T, V>, blocks, 256, 0, s, (const T*)dy, (const T*)z, (T*)dz, npacks);
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "gelu_bwd launch: %s", cudaGetErrorString(e));
}

// partial[blockIdx.y * C + c]
template <typename T, int V, bool GELU>
__global__ void __launch_bounds__(kBgThreads, 4)
bias_grad_kernel(const T* __restrict__ dy, const T* __restrict__ z, T* __restrict__ dz, float* __restrict__ partial,
                 int rows, int C) {
  wait_previous(dy, z);
  const int tx = threadIdx.x % kBgCols, ty = threadIdx.x / kBgCols;
  const int col = (blockIdx.x * kBgCols + tx) * V;
  float acc[V];
#pragma unroll
  for (int k = 0; k < V; ++k) acc[k] = 0.f;
  constexpr int U = GELU ? 2 : 4;                       // rows in flight per thread (63 registers either way)
  const int step = 2 * gridDim.y;
  auto one = [&](const Pack<T, V>& g, const Pack<T, V>& a, size_t at) {
    if (GELU) {
      Pack<T, V> o;
#pragma unroll
      for (int k = 0; k < V; k += 2) {
        float d[2];
        gelu_grad2((float)to_acc<T>(a.v[k]), (float)to_acc<T>(a.v[k + 1]), &d[0], &d[1]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          o.v[k + e] = from_acc<T>((typename AccOf<T>::type)((float)to_acc<T>(g.v[k + e]) * d[e]));
          acc[k + e] += (float)to_acc<T>(o.v[k + e]);   // the sum of what is stored
        }
      }
      st_pack<T, V>(dz + at, o);
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] += (float)to_acc<T>(g.v[k]);
    }
  };
  int r = blockIdx.y * 2 + ty;
  for (; r + (U - 1) * step < rows; r += U * step) {
    Pack<T, V> g[U], a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t at = (size_t)(r + u * step) * C + col;
      g[u] = ld_pack<T, V>(dy + at);
      if (GELU) a[u] = ld_pack<T, V>(z + at);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) one(g[u], a[u], (size_t)(r + u * step) * C + col);
  }
  for (; r < rows; r += step) {
    const size_t at = (size_t)r * C + col;
    Pack<T, V> g = ld_pack<T, V>(dy + at), a;
    if (GELU) a = ld_pack<T, V>(z + at);
    one(g, a, at);
  }
  __shared__ float s[kBgCols][V + 1];
  if (ty == 1) {
#pragma unroll
    for (int k = 0; k < V; ++k) s[tx][k] = acc[k];
  }
  __syncthreads();
  if (ty == 0) {
#pragma unroll
    for (int k = 0; k < V; ++k) partial[(size_t)blockIdx.y * C + col + k] = acc[k] + s[tx][k];
  }
}

// One block per 32 columns; 32 warps each add a contiguous range of the partial rows, then warp 0 adds
// the 32 sums in order: the result does not depend on the launch.
template <typename T>
__global__ void __launch_bounds__(kBgFinCols * kBgFinGroups)
bias_grad_finalize_kernel(const float* __restrict__ partial, int nblocks, int C, T* __restrict__ db) {
  wait_previous(partial);
  const int cx = threadIdx.x % kBgFinCols, grp = threadIdx.x / kBgFinCols;
  const int c = blockIdx.x * kBgFinCols + cx;            // C is a multiple of 32
  const int per = (nblocks + kBgFinGroups - 1) / kBgFinGroups;
  int b = grp * per;
  const int end = min(nblocks, b + per);
  float t = 0.f;
  for (; b + 8 <= end; b += 8) {                        // eight loads in flight, added in row order
    float a[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = partial[(size_t)(b + u) * C + c];
#pragma unroll
    for (int u = 0; u < 8; ++u) t += a[u];
  }
  for (; b < end; ++b) t += partial[(size_t)b * C + c];
  __shared__ float s[kBgFinGroups][kBgFinCols];
  s[grp][cx] = t;
  __syncthreads();
  if (grp == 0) {
    float sum = s[0][cx];
#pragma unroll
    for (int g = 1; g < kBgFinGroups; ++g) sum += s[g][cx];
    db[c] = from_acc<T>((typename AccOf<T>::type)sum);
  }
}

template <typename T>
static int bias_grad_t(const void* dy, const void* z, void* dz, void* db, int rows, int C, void* scratch, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  if (!all_aligned16({dy, z, dz})) return fail(TMPI_ERR_INVALID, "bias_grad: tensors must be 16-byte aligned");
  if (rows < 1 || C % (kBgCols * V)) return fail(TMPI_ERR_UNSUPPORTED, "bias_grad: C=%d must be a multiple of %d", C, kBgCols * V);
  if (z && !dz) return fail(TMPI_ERR_INVALID, "bias_grad: z given without an output for dz");
  const int slabs = C / (kBgCols * V);
  const int per_sm = 4;                                  // resident blocks per SM
  const int rb = std::max(1, std::min((rows + 1) / 2, std::max(1, per_sm * 148 / slabs)));
  const dim3 grid(slabs, rb);
  cudaError_t e = z ? launch_overlapped(bias_grad_kernel<T, V, true>, grid, kBgThreads, 0, s, (const T*)dy, (const T*)z, (T*)dz,
                                        (float*)scratch, rows, C)
                    : launch_overlapped(bias_grad_kernel<T, V, false>, grid, kBgThreads, 0, s, (const T*)dy, (const T*)nullptr, (T*)nullptr,
                                        (float*)scratch, rows, C);
  if (e == cudaSuccess)
    e = launch_overlapped(bias_grad_finalize_kernel<T>, C / kBgFinCols, kBgFinCols * kBgFinGroups, 0, s, (const float*)scratch, rb, C, (T*)db);
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "bias_grad launch: %s", cudaGetErrorString(e));
}

}  // namespace tmpi

using namespace tmpi;

extern "C" {

size_t tmpi_bias_grad_scratch_bytes(int channels) { return (size_t)kBgMaxRowBlocks * channels * sizeof(float); }

// db[c] = sum_r dz[r, c] with dz = dy * gelu'(z) written to `dz` when z is given, else dz = dy (nothing written).
// dy, z, dz: [rows, channels]; db: [channels]; all of `dtype`.
int tmpi_bias_grad(const void* dy, const void* z, void* dz, void* db, int rows, int channels, int dtype, void* scratch,
                   void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return bias_grad_t<__nv_bfloat16>(dy, z, dz, db, rows, channels, scratch, s);
    case TMPI_F16: return bias_grad_t<__half>(dy, z, dz, db, rows, channels, scratch, s);
    case TMPI_F32: return bias_grad_t<float>(dy, z, dz, db, rows, channels, scratch, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "bias_grad: dtype %d", dtype);
}

// dz = dy * gelu'(z) for n elements of `dtype`.
int tmpi_gelu_bwd(const void* dy, const void* z, void* dz, size_t n, int dtype, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return gelu_bwd_t<__nv_bfloat16>(dy, z, dz, n, s);
    case TMPI_F16: return gelu_bwd_t<__half>(dy, z, dz, n, s);
    case TMPI_F32: return gelu_bwd_t<float>(dy, z, dz, n, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "gelu_bwd: dtype %d", dtype);
}

// y = gelu(z) (erf form) for n elements of `dtype`; the forward companion of tmpi_bias_grad's derivative.
int tmpi_gelu_fwd(const void* z, void* y, size_t n, int dtype, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  switch (dtype) {
    case TMPI_BF16: return gelu_fwd_t<__nv_bfloat16>(z, y, n, s);
    case TMPI_F16: return gelu_fwd_t<__half>(z, y, n, s);
    case TMPI_F32: return gelu_fwd_t<float>(z, y, n, s);
  }
  return fail(TMPI_ERR_UNSUPPORTED, "gelu_fwd: dtype %d", dtype);
}

}  // extern "C"
