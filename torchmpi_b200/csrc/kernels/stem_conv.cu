// The ResNet stem convolution (7 x 7, stride 2, pad 3, 3 input channels, 64 output channels) as an implicit GEMM on the
// tcgen05 tensor cores: forward and weight gradient, without a patch matrix.
//
// The input goes to shared memory as rows of 16-byte units, one per pair of pixels (2p, 2p + 1), each pixel padded to four
// channels.  The window of output pixel ow covers the four pairs ow - 2 .. ow + 1 (one padded tap on the left), so
// neighbouring output pixels read neighbouring units, and a row of units IS the operand in the unswizzled core-matrix
// layout of the tensor core: eight consecutive output pixels x 8 values are 128 contiguous bytes, the next tap pair is the
// same 128 bytes moved by one unit.  Overlapping core matrices cost nothing, so nothing is copied per window.
//
//   forward          Y[ow, co] += X[ow, (pair, channel)] W[co, (pair, channel)] for each input row of a window, two output rows
//                    at a time: input rows 2 - 6 of the nine that they cover meet kernel row r for the first and r - 2 for
//                    the second, side by side in one operand of 128 columns: 19 MMAs of 128 x 128 (or 64) x 16 for two rows
//                    (K = 7 rows x 4 pairs x 8 = 224 for 147 weights) in place of 28 narrow ones.  An MMA is paced by its
//                    128-row operand, so a wide one costs little more: with the pooling stage, forward and backward,
//                    770 -> 757 us at 256 x 224 x 224, of which this kernel takes about 125 (138 before).
//   weight gradient  the output pixels are the K dimension.  Two output rows share an operand: M = 128 = dY rows (i, i + 1)
//                    of 64 channels, N = 80 = ten input rows x 8 values of one tap pair (the rows are a constant stride
//                    apart), four MMAs per 16 pixels; input row r meets kernel row r of dY row i and r - 2 of row i + 1.
//                    Partial sums per CTA, added in CTA order by a second kernel (deterministic).
//                    Where K or M is padded (an output width that is not a multiple of 16, the last row of an odd height) dY is
//                    zero and the image is not: the operands there are arranged so that a non-finite pixel meets no zero
//                    that is not its own (tail units, the single row).
//
// What bounds it: forward the 411 MB of output (62 us at the copy rate, 256 images of 224 x 224) and, about as much, the
// MMAs; the weight gradient the reads of dY, the same bytes, and the MMAs (their 128-row dY
// operand comes out of shared memory once per tap pair).  The patch matrix that both products read before was 1.03 GB,
// written once and read twice.  Measured, 256 x 224 x 224: forward about 125 us
// (patch matrix 354 + product 262 + weight layout 9), weight gradient 147 us (split-K product 221).
//
// The reference has no convolution of its own (it trains Torch7 modules).  One persistent CTA per SM, work in chunks of
// eight output rows, double-buffered; every wait is bounded.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <mutex>
#include "sm100_ptx.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"

namespace tmpi {

int gemm_sm_count();
int* gemm_status_word();
int make_tmap_bf16_4d(CUtensorMap* map, const void* base, const uint64_t (&dims)[4], const uint32_t (&box)[4]);

namespace stem {

constexpr int COUT = 64, TAPS = 4, KROWS = 7, R = 8, IN_ROWS = 2 * R + 6;      // chunk: R output rows, 2 R + 5 input rows (+ 1: N = 80)
constexpr int MAX_OW = 128;
constexpr int LOADERS = 256, THREADS = 512;        // warp 0 issues MMAs, warps 4-7 drain, warps 8-15 load x; wgrad: warp 1 loads dY
constexpr int STAGING = 4096;                      // 32 pixels x 64 channels
constexpr int W_BYTES = KROWS * TAPS * 8 * COUT * 2;
constexpr int W_BLOCK = COUT * 16, W_TAP = KROWS * W_BLOCK;      // one kernel row of a tap pair, one tap pair
constexpr int ACCS = 4, DY_STAGES = 3, WG_N = 80;
constexpr int TAILS = 2;                           // tap pairs whose last 16 pixels are kept once more
constexpr int SINGLE_N = 32, SINGLE_COL = TAPS * WG_N;      // accumulators of an odd height's last row: input rows 2..5 of each tap pair
constexpr unsigned long long kWaitBudgetNs = 4000000000ull;

struct Shared {
  uint64_t x_full[2], x_empty[2], acc_full[ACCS], acc_empty[ACCS], dy_full[DY_STAGES], dy_empty[DY_STAGES];
  uint32_t tmem_base;
  int error;
};

struct Params {
  int N, H, W, OH, OW, ow16, units, chunks_per_image, chunks;
  int row_bytes;               // shared-memory bytes of one input row: units * 16 (+ the tail units, see load_rows)
  int64_t ws_co, ws_c, ws_h, ws_w;      // strides of the weight (and its gradient), elements
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;
  float* partial;              // weight gradient: [gridDim.x][128][TAPS * WG_N]
  int* status;
};

__device__ __forceinline__ void fail(Shared* sh, const Params& p, int where) {
  atomicExch(&sh->error, where);
  if (p.status) atomicCAS(p.status, 0, 1000 + where);
}
#define STEM_WAIT(bar, parity, where) \
  do { if (!sm100::mbar_wait((bar), (parity), kWaitBudgetNs) || sh->error) { fail(sh, p, (where)); return; } } while (0)

// Unswizzled operand: core matrices of 8 rows x 16 bytes, 128 contiguous bytes each.  K-major: `lead` between the two
// core matrices along K, `stride` between groups of eight rows.  MN-major: `stride` between core matrices along M / N,
// `lead` between groups of eight along K.
__device__ __forceinline__ uint64_t desc_plain(uint32_t addr, uint32_t lead, uint32_t stride) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(lead >> 4) << 16 | (uint64_t)(stride >> 4) << 32 | (uint64_t)1 << 46;
}

__device__ __forceinline__ bool chunk(const Params& p, int it, int* n, int* oh0) {
  const int c = blockIdx.x + it * gridDim.x;
  if (c >= p.chunks) return false;
  *n = c / p.chunks_per_image;
  *oh0 = (c - *n * p.chunks_per_image) * R;
  return true;
}

// Warps 8-15: the input rows of a chunk as units.  A unit is 12 contiguous bytes of the image (W is even: a pair is inside
// or outside as a whole).  Four units per thread are in flight; the loads of a chunk's first four start before the buffer
// is free.
// TAIL (weight gradient): where the output width is not a multiple of 16, the last 16 output pixels of a row are partly padding,
// and under the first two tap pairs the padding's windows would reach into the image.  Each row carries those 16 units once
// more per tap pair, zeros (written at the start) where the output pixel is padding.
template <bool TAIL>
__device__ void load_rows(Shared* sh, unsigned char* rows, const Params& p, int tid) {
  const int total = IN_ROWS * p.units, pairs = p.W / 2;
  int n, oh0;
  for (int it = 0; chunk(p, it, &n, &oh0); ++it) {
    const int b = it & 1;
    unsigned char* dst = rows + b * IN_ROWS * p.row_bytes;
    const uint32_t* img = reinterpret_cast<const uint32_t*>(p.x) + (size_t)n * p.H * (p.W * 3 / 2);
    bool free = it < 2;
    for (int t0 = tid; t0 < total; t0 += 4 * LOADERS) {
      uint32_t w[4][3];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = t0 + q * LOADERS;
        const int row = t / p.units, pr = t - row * p.units - 2, ih = 2 * oh0 - 3 + row;
        w[q][0] = w[q][1] = w[q][2] = 0u;
        if (t < total && ih >= 0 && ih < p.H && pr >= 0 && pr < pairs) {
          const uint32_t* s = img + (size_t)ih * (p.W * 3 / 2) + pr * 3;
          w[q][0] = __ldg(s); w[q][1] = __ldg(s + 1); w[q][2] = __ldg(s + 2);
        }
      }
      if (!free) { STEM_WAIT(&sh->x_empty[b], ((it >> 1) - 1) & 1, 61); free = true; }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int t = t0 + q * LOADERS;
        if (t >= total) continue;
        const uint4 unit = make_uint4(w[q][0], w[q][1] & 0xffffu, (w[q][1] >> 16) | (w[q][2] << 16), w[q][2] >> 16);
        if constexpr (!TAIL) {
          *reinterpret_cast<uint4*>(dst + (size_t)t * 16) = unit;
        } else {
          const int row = t / p.units, u = t - row * p.units, rest = p.OW & 15;
          unsigned char* line = dst + (size_t)row * p.row_bytes;
          *reinterpret_cast<uint4*>(line + u * 16) = unit;
#pragma unroll
          for (int tap = 0; tap < TAILS; ++tap) {
            const int j = u - (p.OW - rest) - tap;               // pixel among the last 16
            if (j >= 0 && j < rest) *reinterpret_cast<uint4*>(line + (p.units + tap * 16 + j) * 16) = unit;
          }
        }
      }
    }
    sm100::fence_proxy_async_smem();
    __syncwarp();
    if ((tid & 31) == 0) sm100::mbar_arrive(&sh->x_full[b]);
  }
}

__device__ __forceinline__ void setup(Shared* sh, int warp) {
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) { sm100::mbar_init(&sh->x_full[b], LOADERS / 32); sm100::mbar_init(&sh->x_empty[b], 1); }
    for (int a = 0; a < ACCS; ++a) { sm100::mbar_init(&sh->acc_full[a], 1); sm100::mbar_init(&sh->acc_empty[a], 4); }
    for (int s = 0; s < DY_STAGES; ++s) { sm100::mbar_init(&sh->dy_full[s], 1); sm100::mbar_init(&sh->dy_empty[s], 1); }
    sh->error = 0;
    sm100::fence_barrier_init();
  }
  if (warp == 0) {
    sm100::tmem_alloc(&sh->tmem_base, 512);
    sm100::tmem_relinquish();
  }
}
__device__ __forceinline__ void teardown(Shared* sh, int warp) {
  __syncwarp();
  sm100::tc_fence_before();
  __syncthreads();
  if (sh->error && threadIdx.x == 0) {
    const unsigned long long t0 = sm100::now_ns();
    while (sm100::now_ns() - t0 < 200000000ull) { __nanosleep(1000); }   // copies in flight land within microseconds
  }
  __syncthreads();
  if (warp == 0) {
    sm100::tc_fence_after();
    sm100::tmem_dealloc(sh->tmem_base, 512);
  }
}

// ---------------------------------------------------------------- forward
// Weights of a tap pair: a block of 64 output channels x 16 bytes per kernel row, in the order 6 4 2 0 5 3 1, so that the
// block of row r is followed by that of row r - 2.
__device__ __forceinline__ int weight_block(int kh) { return (kh & 1) ? 4 + (5 - kh) / 2 : (6 - kh) / 2; }

__device__ void fwd_mma(Shared* sh, unsigned char* rows, unsigned char* weights, const Params& p) {
  constexpr uint32_t idesc_one = sm100::make_idesc_f16(128, COUT, true), idesc_two = sm100::make_idesc_f16(128, 2 * COUT, true);
  const uint32_t x0 = sm100::smem_u32(rows), w0 = sm100::smem_u32(weights);
  int n, oh0, count = 0;
  for (int it = 0; chunk(p, it, &n, &oh0); ++it) {
    const int b = it & 1;
    STEM_WAIT(&sh->x_full[b], (it >> 1) & 1, 62);
    const int lines = min(R, p.OH - oh0);
    for (int i = 0; i < lines; i += 2, ++count) {
      const int acc = count % ACCS;
      if (count >= ACCS) STEM_WAIT(&sh->acc_empty[acc], (count / ACCS - 1) & 1, 63);
      sm100::tc_fence_after();
      const bool two = i + 1 < lines;
      const uint32_t d = sh->tmem_base + acc * 2 * COUT;
#pragma unroll
      for (int r = 0; r < KROWS + 2; ++r) {                  // input row; tap pairs 2 h and the next
        if (r >= KROWS && !two) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint64_t a = desc_plain(x0 + (uint32_t)(b * IN_ROWS + 2 * i + r) * p.row_bytes + h * 32, 16, 128);
          const uint32_t w = w0 + h * 2 * W_TAP + weight_block(r < KROWS ? r : r - 2) * W_BLOCK;
          // rows 0 and 1 are the first output row's alone, 7 and 8 the second one's, whose sums start at row 2
          if (r == 2 && h == 0 && two) {
            sm100::umma_f16(d, a, desc_plain(w, W_TAP, 128), idesc_one, 1u);
            sm100::umma_f16(d + COUT, a, desc_plain(w + W_BLOCK, W_TAP, 128), idesc_one, 0u);
          } else {
            sm100::umma_f16(r < KROWS ? d : d + COUT, a, desc_plain(w, W_TAP, 128), two && r >= 2 && r < KROWS ? idesc_two : idesc_one,
                            (r | h) ? 1u : 0u);
          }
        }
      }
      sm100::umma_commit(&sh->acc_full[acc]);
    }
    sm100::umma_commit(&sh->x_empty[b]);
  }
}

// The padded tap multiplies the pixel left of the window by a weight of zero, which is NaN in all channels when that pixel is
// not finite.  A pixel whose first channel came out NaN is looked at again, and computed without that tap if it was the
// reason: 147 x 64 multiply-adds on one thread, reached by non-finite images only.
__device__ __noinline__ void redo_pixel(const __nv_bfloat16* img, int H, int W, const unsigned char* weights, unsigned char* out,
                                        int swizzle, int oh, int ow) {
  const int iw0 = 2 * ow - 3;
  bool pad = false;
  for (int kh = 0; kh < KROWS && iw0 > 0; ++kh) {
    const int ih = 2 * oh - 3 + kh;
    for (int c = 0; c < 3 && ih >= 0 && ih < H; ++c) pad |= !isfinite(__bfloat162float(img[((size_t)ih * W + iw0 - 1) * 3 + c]));
  }
  if (!pad) return;
  const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(weights);
#pragma unroll 1
  for (int co = 0; co < COUT; ++co) {
    float sum = 0.f;
#pragma unroll 1
    for (int kh = 0; kh < KROWS; ++kh) {
      const int ih = 2 * oh - 3 + kh;
      if (ih < 0 || ih >= H) continue;
      for (int kw = 0; kw < 7; ++kw) {
        if (iw0 + kw < 0 || iw0 + kw >= W) continue;
        for (int c = 0; c < 3; ++c)
          sum += __bfloat162float(img[((size_t)ih * W + iw0 + kw) * 3 + c]) *
                 __bfloat162float(w[(((kw + 1) / 2 * KROWS + weight_block(kh)) * COUT + co) * 8 + ((kw + 1) & 1) * 4 + c]);
      }
    }
    *reinterpret_cast<__nv_bfloat16*>(out + (((co >> 3) ^ swizzle) << 4) + (co & 7) * 2) = __float2bfloat16(sum);
  }
}

__device__ void fwd_drain(Shared* sh, unsigned char* staging, const unsigned char* weights, const Params& p, const CUtensorMap* my, int quarter, int lane) {
  const uint32_t tm = sh->tmem_base + ((uint32_t)(quarter * 32) << 16);
  int n, oh0, count = 0, row = 0;                             // accumulators and rows drained
  for (int it = 0; chunk(p, it, &n, &oh0); ++it) {
    const int lines = min(R, p.OH - oh0);
    for (int i = 0; i < lines; ++i, ++row) {
      const int acc = count % ACCS;
      const bool second = i & 1, last = second || i + 1 == lines;            // of its accumulator
      if (!second) {
        STEM_WAIT(&sh->acc_full[acc], (count / ACCS) & 1, 64);
        sm100::tc_fence_after();
      }
      uint32_t r[2][32];
      const uint32_t at = tm + acc * 2 * COUT + (second ? COUT : 0);
      sm100::tmem_ld_32x32(at, r[0]);
      sm100::tmem_ld_32x32(at + 32, r[1]);
      sm100::tmem_ld_wait();
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (last) sm100::mbar_arrive(&sh->acc_empty[acc]);
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the store two rows ago has read its tile
      }
      __syncwarp();
      if (quarter * 32 < p.OW) {
        unsigned char* stg = staging + (quarter * 2 + (row & 1)) * STAGING;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int j = (u & 3) * 8 + 2 * e;
            __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[u >> 2][j]), __uint_as_float(r[u >> 2][j + 1]));
            w[e] = *reinterpret_cast<uint32_t*>(&h);
          }
          *reinterpret_cast<uint4*>(stg + lane * 128 + ((u ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (isnan(__uint_as_float(r[0][0])) && quarter * 32 + lane < p.OW)
          redo_pixel(p.x + (size_t)n * p.H * p.W * 3, p.H, p.W, weights, stg + lane * 128, lane & 7, oh0 + i, quarter * 32 + lane);
        sm100::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) sm100::tma_store_4d(my, stg, 0, quarter * 32, oh0 + i, n);      // pixels beyond the row are clipped
      }
      if (lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      if (last) ++count;
    }
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

__global__ void __launch_bounds__(THREADS, 1) stem_fwd_kernel(const __grid_constant__ CUtensorMap map_y, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* staging = smem;                              // 4 warps x 2 tiles
  unsigned char* weights = smem + 8 * STAGING;
  unsigned char* rows = weights + W_BYTES;
  // the 128-row operand of the last input row runs on past it by up to MAX_OW units, into the tail that follows the rows
  Shared* sh = (Shared*)(rows + 2 * IN_ROWS * p.row_bytes + (MAX_OW + 4) * 16);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  setup(sh, warp);
  for (int t = threadIdx.x; t < KROWS * TAPS * COUT; t += THREADS) {
    const int co = t % COUT, unit = t / COUT, kh = unit / TAPS, tap = unit % TAPS;
    unsigned short v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int kw = 2 * tap + (e >> 2) - 1, c = e & 3;
      v[e] = 0;
      if (kw >= 0 && kw < 7 && c < 3)
        v[e] = *reinterpret_cast<const unsigned short*>(p.w + co * p.ws_co + c * p.ws_c + kh * p.ws_h + kw * p.ws_w);
    }
    *reinterpret_cast<uint4*>(weights + tap * W_TAP + weight_block(kh) * W_BLOCK + co * 16) =
        make_uint4(v[0] | (uint32_t)v[1] << 16, v[2] | (uint32_t)v[3] << 16, v[4] | (uint32_t)v[5] << 16, v[6] | (uint32_t)v[7] << 16);
  }
  sm100::fence_proxy_async_smem();
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  if (warp == 0) {
    if (sm100::elect_one()) fwd_mma(sh, rows, weights, p);
  } else if (warp >= 8) {
    load_rows<false>(sh, rows, p, threadIdx.x - 256);
  } else if (warp >= 4) {
    fwd_drain(sh, staging, weights, p, &map_y, warp & 3, lane);
  }
  teardown(sh, warp);
}

// ---------------------------------------------------------------- weight gradient
// PADDED: an output width that is not a multiple of 16 or an odd output height (see load_rows and the row alone below).  The
// other form stays as it is where nothing is padded: its code is shorter, and the thread that issues the MMAs is paced by it.
// 256 x 200 x 200 135 us, 256 x 222 x 224 152 (136 and 148 without the precautions), 256 x 224 x 224, not padded, 148.
template <bool PADDED>
__global__ void __launch_bounds__(THREADS, 1) stem_wgrad_kernel(const __grid_constant__ CUtensorMap map_dy, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int dy_row = p.ow16 * 128, dy_stage = 2 * dy_row;     // a pair of dY rows of 64 channels, 128-byte swizzle
  unsigned char* dys = smem;
  unsigned char* rows = smem + DY_STAGES * dy_stage;
  Shared* sh = (Shared*)(rows + 2 * IN_ROWS * p.row_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  setup(sh, warp);
  if constexpr (PADDED) {
    for (int t = threadIdx.x; t < 2 * IN_ROWS * TAILS * 16; t += THREADS)
      *reinterpret_cast<uint4*>(rows + (t / (TAILS * 16)) * p.row_bytes + (p.units + t % (TAILS * 16)) * 16) = make_uint4(0u, 0u, 0u, 0u);
    sm100::fence_proxy_async_smem();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  if constexpr (PADDED) {                                     // two kinds of products, either may come first: all sums start at zero
    if (warp >= 4 && warp < 8) {
      const uint32_t zero[16] = {};
      for (int c = 0; c < SINGLE_COL + TAPS * SINGLE_N; c += 16) sm100::tmem_st_32x16(sh->tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c, zero);
      sm100::tmem_st_wait();
    }
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
  }
  int n, oh0;
  if (warp >= 8) {
    load_rows<PADDED>(sh, rows, p, threadIdx.x - 256);
  } else if (warp == 1) {
    if (sm100::elect_one()) [&]() {
      int count = 0;
      for (int it = 0; chunk(p, it, &n, &oh0); ++it)
        for (int i = 0; i < R && oh0 + i < p.OH; i += 2, ++count) {
          const int s = count % DY_STAGES;
          if (count >= DY_STAGES) STEM_WAIT(&sh->dy_empty[s], (count / DY_STAGES - 1) & 1, 65);
          sm100::mbar_expect_tx(&sh->dy_full[s], dy_stage);
          // rows beyond the image and pixels beyond the row are zeros
          sm100::tma_load_4d(dys + s * dy_stage, &map_dy, 0, 0, oh0 + i, n, &sh->dy_full[s]);
          sm100::tma_load_4d(dys + s * dy_stage + dy_row, &map_dy, 0, 0, oh0 + i + 1, n, &sh->dy_full[s]);
        }
    }();
  } else if (warp == 0) {
    if (sm100::elect_one()) [&]() {
      constexpr uint32_t idesc = sm100::make_idesc_f16(128, WG_N, true, true, true);      // both operands MN-major (pixels are K)
      constexpr uint32_t idesc_16 = sm100::make_idesc_f16(128, 16, true, true, true);
      constexpr uint32_t idesc_single = sm100::make_idesc_f16(128, SINGLE_N, true, true, true);
      const uint32_t x0 = sm100::smem_u32(rows);
      int count = 0;
      for (int it = 0; chunk(p, it, &n, &oh0); ++it) {
        const int b = it & 1;
        STEM_WAIT(&sh->x_full[b], (it >> 1) & 1, 66);
        for (int i = 0; i < R && oh0 + i < p.OH; i += 2, ++count) {
          const int s = count % DY_STAGES;
          STEM_WAIT(&sh->dy_full[s], (count / DY_STAGES) & 1, 67);
          sm100::tc_fence_after();
          const uint64_t a = sm100::make_desc_sw128_mn(sm100::smem_u32(dys + s * dy_stage), dy_row, 1024);
          const uint32_t x_row = x0 + (uint32_t)(b * IN_ROWS + 2 * i) * p.row_bytes;
          if constexpr (!PADDED) {
            for (int k = 0; k < p.ow16 / 16; ++k)
#pragma unroll
              for (int t = 0; t < TAPS; ++t)
                sm100::umma_f16(sh->tmem_base + t * WG_N, a + (uint64_t)((k * 16 * 128) >> 4), desc_plain(x_row + (k * 16 + t) * 16, 128, p.row_bytes),
                                idesc, (count | k) ? 1u : 0u);
          } else {
            // descriptors advance by units of 16 bytes in their address field
            const uint64_t x = desc_plain(x_row, 128, p.row_bytes), x2 = desc_plain(x_row + 2 * p.row_bytes, 128, p.row_bytes);
            const int blocks = p.OW / 16;                        // of 16 whole pixels
            auto block = [&](int k, int (&at)[TAPS]) {
              if (oh0 + i + 1 < p.OH) {
#pragma unroll
                for (int t = 0; t < TAPS; ++t) sm100::umma_f16(sh->tmem_base + t * WG_N, a + (uint64_t)(k * 128), x + (uint64_t)at[t], idesc, 1u);
              } else {
                // Row i alone: dY row i + 1 is padding.  Its products land in the other 64 accumulator rows: input rows 0 and 1
                // are none of its, input rows 2 - 5 go to columns of their own, later ones lie below the image.
#pragma unroll
                for (int t = 0; t < TAPS; ++t) {
                  sm100::umma_f16(sh->tmem_base + t * WG_N, a + (uint64_t)(k * 128), x + (uint64_t)at[t], idesc_16, 1u);
                  sm100::umma_f16(sh->tmem_base + SINGLE_COL + t * SINGLE_N, a + (uint64_t)(k * 128), x2 + (uint64_t)at[t], idesc_single, 1u);
                }
              }
            };
            for (int k = 0; k < blocks; ++k) {
              int at[TAPS] = {k * 16, k * 16 + 1, k * 16 + 2, k * 16 + 3};
              block(k, at);
            }
            if (p.OW & 15) {                                     // the cut last block: tail units under the first tap pairs
              int at[TAPS] = {p.units, p.units + 16, blocks * 16 + 2, blocks * 16 + 3};
              block(blocks, at);
            }
          }
          sm100::umma_commit(&sh->dy_empty[s]);
        }
        sm100::umma_commit(&sh->x_empty[b]);
      }
      sm100::umma_commit(&sh->acc_full[0]);
    }();
  } else if (warp >= 4) {
    [&]() {
      STEM_WAIT(&sh->acc_full[0], 0, 68);
      sm100::tc_fence_after();
      const int row = (warp & 3) * 32 + lane;
      const uint32_t tm = sh->tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
      float* out = p.partial + ((size_t)blockIdx.x * 128 + row) * (TAPS * WG_N);
      for (int c = 0; c < TAPS * WG_N; c += 32) {
        uint32_t r[32];
        sm100::tmem_ld_32x32(tm + c, r);
        sm100::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(out + c + j) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                                                __uint_as_float(r[j + 3]));
      }
      if (PADDED && (warp & 3) < 2) {                           // the first 64 rows: the single rows' sums on top
        for (int t = 0; t < TAPS; ++t) {
          uint32_t r[32];
          sm100::tmem_ld_32x32(tm + SINGLE_COL + t * SINGLE_N, r);
          sm100::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            float4* o = reinterpret_cast<float4*>(out + t * WG_N + 16 + j);
            const float4 v = *o;
            *o = make_float4(v.x + __uint_as_float(r[j]), v.y + __uint_as_float(r[j + 1]), v.z + __uint_as_float(r[j + 2]),
                             v.w + __uint_as_float(r[j + 3]));
          }
        }
      }
      sm100::tc_fence_before();
    }();
  }
  teardown(sh, warp);
}

// One block per output channel and tap pair: 32 groups of threads add the partial rows of a contiguous range of CTAs (dY row i and,
// ten input rows being shared by two dY rows, row i + 1 two input rows further on), all loads of a thread in flight; the groups' sums are
// added in order.  Bound by the 24 MB of partial sums.  A block per channel, with ten groups, 7.7 us; now 6.0.
constexpr int RED_COLS = WG_N / 4, RED_GROUPS = 32, RED_ROWS = 5;
__global__ void __launch_bounds__(RED_COLS * RED_GROUPS)
stem_wgrad_reduce_kernel(const float* __restrict__ partial, int ctas, __nv_bfloat16* __restrict__ dw, int64_t s_co, int64_t s_c, int64_t s_h,
                         int64_t s_w) {
  __shared__ float4 sum[RED_GROUPS][2][RED_COLS];
  const int col = threadIdx.x % RED_COLS, grp = threadIdx.x / RED_COLS, co = blockIdx.x, tap = blockIdx.y;
  const int per = (ctas + RED_GROUPS - 1) / RED_GROUPS, end = min(ctas, (grp + 1) * per);
  float4 a[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  for (int c0 = grp * per; c0 < end; c0 += RED_ROWS) {
    float4 v[RED_ROWS][2];
#pragma unroll
    for (int r = 0; r < RED_ROWS; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        v[r][h] = c0 + r < end ? __ldg(reinterpret_cast<const float4*>(partial + ((size_t)(c0 + r) * 128 + h * 64 + co) * (TAPS * WG_N) + tap * WG_N) + col)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < RED_ROWS; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) { a[h].x += v[r][h].x; a[h].y += v[r][h].y; a[h].z += v[r][h].z; a[h].w += v[r][h].w; }
  }
  sum[grp][0][col] = a[0];
  sum[grp][1][col] = a[1];
  __syncthreads();
  for (int o = threadIdx.x; o < 147; o += blockDim.x) {
    const int kh = o / 21, kw = o % 21 / 3, c = o % 3, e = (kw + 1) & 1;
    if (((kw + 1) >> 1) != tap) continue;
    const int at0 = kh * 8 + e * 4 + c, at1 = at0 + 16;
    float t = 0.f;
#pragma unroll
    for (int g = 0; g < RED_GROUPS; ++g)
      t += reinterpret_cast<const float*>(sum[g][0])[at0] + reinterpret_cast<const float*>(sum[g][1])[at1];
    dw[co * s_co + c * s_c + kh * s_h + kw * s_w] = __float2bfloat16_rn(t);
  }
}

static int fill(Params* p, const void* x, int N, int H, int W, int cout, const int64_t* strides) {
  if (N < 1 || H < 1 || W < 8) return tmpi::fail(TMPI_ERR_INVALID, "stem convolution: empty input");
  const int OH = (H - 1) / 2 + 1, OW = (W - 1) / 2 + 1;
  if (cout != COUT || W % 8 || OW > MAX_OW || ((uintptr_t)x & 15))
    return tmpi::fail(TMPI_ERR_UNSUPPORTED, "stem convolution: needs %d output channels, W a multiple of 8 up to %d and a 16-byte aligned input", COUT, 2 * MAX_OW);
  p->N = N; p->H = H; p->W = W; p->OH = OH; p->OW = OW;
  p->ow16 = (OW + 15) / 16 * 16;
  p->units = p->ow16 + 4;
  p->row_bytes = p->units * 16;
  p->chunks_per_image = (OH + R - 1) / R;
  if ((int64_t)N * p->chunks_per_image > 0x7fffffffLL) return tmpi::fail(TMPI_ERR_UNSUPPORTED, "stem convolution: too many images");
  p->chunks = N * p->chunks_per_image;
  p->x = (const __nv_bfloat16*)x;
  p->ws_co = strides[0]; p->ws_c = strides[1]; p->ws_h = strides[2]; p->ws_w = strides[3];
  p->status = gemm_status_word();
  return TMPI_OK;
}

}  // namespace stem
}  // namespace tmpi

using namespace tmpi;

extern "C" {

// 1 if tmpi_stem_conv_fwd / _wgrad take an image width and a number of output channels
int tmpi_stem_conv_supported(int W, int cout) { return cout == stem::COUT && W >= 8 && W % 8 == 0 && (W - 1) / 2 + 1 <= stem::MAX_OW; }

// y[N, OH, OW, 64] (channels-last) = convolution of x [N, H, W, 3] (channels-last) with w [64, 3, 7, 7] (any strides, given in
// elements), stride 2, pad 3.  bf16, fp32 accumulation.
int tmpi_stem_conv_fwd(const void* x, const void* w, void* y, int N, int H, int W, int cout, const int64_t* w_strides, void* stream) {
  stem::Params p{};
  int st = stem::fill(&p, x, N, H, W, cout, w_strides);
  if (st) return st;
  p.w = (const __nv_bfloat16*)w;
  CUtensorMap my;
  if ((st = make_tmap_bf16_4d(&my, y, {(uint64_t)stem::COUT, (uint64_t)p.OW, (uint64_t)p.OH, (uint64_t)N}, {64, 32, 1, 1}))) return st;
  const int smem = 8 * stem::STAGING + stem::W_BYTES + 2 * stem::IN_ROWS * p.row_bytes + (stem::MAX_OW + 4) * 16 + (int)sizeof(stem::Shared);
  cudaError_t e = cudaFuncSetAttribute(stem::stem_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return fail(TMPI_ERR_CUDA, "stem convolution: shared memory attribute: %s", cudaGetErrorString(e));
  stem::stem_fwd_kernel<<<std::min(p.chunks, gemm_sm_count()), stem::THREADS, smem, (cudaStream_t)stream>>>(my, p);
  e = cudaGetLastError();
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "stem convolution launch: %s", cudaGetErrorString(e));
}

size_t tmpi_stem_conv_wgrad_workspace_bytes(void) { return (size_t)gemm_sm_count() * 128 * stem::TAPS * stem::WG_N * sizeof(float); }

// dw [64, 3, 7, 7] (strides as given) from dy [N, OH, OW, 64] and x; workspace: tmpi_stem_conv_wgrad_workspace_bytes.
int tmpi_stem_conv_wgrad(const void* dy, const void* x, void* dw, int N, int H, int W, int cout, const int64_t* w_strides,
                         void* workspace, size_t workspace_bytes, void* stream) {
  stem::Params p{};
  int st = stem::fill(&p, x, N, H, W, cout, w_strides);
  if (st) return st;
  const int grid = std::min(p.chunks, gemm_sm_count());
  if (workspace_bytes < (size_t)grid * 128 * stem::TAPS * stem::WG_N * sizeof(float))
    return fail(TMPI_ERR_INVALID, "stem convolution: the workspace is too small");
  p.partial = (float*)workspace;
  CUtensorMap mdy;
  if ((st = make_tmap_bf16_4d(&mdy, dy, {(uint64_t)stem::COUT, (uint64_t)p.OW, (uint64_t)p.OH, (uint64_t)N}, {64, (uint32_t)p.ow16, 1, 1}))) return st;
  const bool padded = p.OW % 16 != 0 || p.OH % 2 != 0;
  if (padded) p.row_bytes += stem::TAILS * 16 * 16;
  const int smem = stem::DY_STAGES * 2 * p.ow16 * 128 + 2 * stem::IN_ROWS * p.row_bytes + (int)sizeof(stem::Shared);
  const auto kernel = padded ? stem::stem_wgrad_kernel<true> : stem::stem_wgrad_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return fail(TMPI_ERR_CUDA, "stem weight gradient: shared memory attribute: %s", cudaGetErrorString(e));
  kernel<<<grid, stem::THREADS, smem, (cudaStream_t)stream>>>(mdy, p);
  stem::stem_wgrad_reduce_kernel<<<dim3(stem::COUT, stem::TAPS), stem::RED_COLS * stem::RED_GROUPS, 0, (cudaStream_t)stream>>>(
      (const float*)workspace, grid, (__nv_bfloat16*)dw, p.ws_co, p.ws_c, p.ws_h, p.ws_w);
  e = cudaGetLastError();
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "stem weight gradient launch: %s", cudaGetErrorString(e));
}

}  // extern "C"
