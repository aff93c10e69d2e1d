// bf16 GEMM on CTA pairs: C[M,N] = act(A[M,K] * B[N,K]^T + bias) with 256 x 256 tiles computed by
// two CTAs of a cluster (gemm_pair.cuh).  One cluster per TPC, persistent.
#include "gemm_pair.cuh"
#include "pdl.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"
#include <algorithm>
#include <cstring>
#include <mutex>

namespace tmpi {

int make_tmap_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
int gemm_sm_count();

namespace gemm2 {

// p.tiles_m counts 256-row tiles here.  WITH_GELU: gelu(C) goes to map_y beside C.
template <int MODE>
__global__ void __launch_bounds__(GROUP_THREADS, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_y, const Problem p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *tiles, *staging;
  Shared* sh;
  constexpr int NST = MODE == WITH_GELU ? STAGES - 1 : STAGES;
  carve<NST>(smem_raw, &tiles, &sh, &staging);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = sm100::cluster_ctarank();
  setup(sh, warp, &map_a, &map_b, 4 * GROUPS);
  const __nv_bfloat16 *bias = p.bias, *residual = p.residual;      // read through the read-only path: not before the wait (pdl.cuh)
  wait_previous(bias, residual);

  const int total = p.tiles_m * p.tiles_n;
  const int cluster = blockIdx.x >> 1, nclusters = gridDim.x >> 1;
  auto order = [&](int it, int* m_blk, int* n_blk) -> bool {
    const int t = cluster + it * nclusters;
    if (t >= total) return false;
    int m_tile;
    band_order(t, p.tiles_m, p.tiles_n, &m_tile, n_blk);
    *m_blk = m_tile * 2 + (int)rank;
    return true;
  };
  if (warp == 0) {
    if (sm100::elect_one()) producer<NST>(sh, tiles, p, &map_a, &map_b, rank, order, [](int, const CUtensorMap**, int*) { return true; });
  } else if (warp == 1) {
    if (rank == 0 && sm100::elect_one()) mma_issuer<NST>(sh, tiles, p, order);
  } else {
    epilogue_groups<MODE>(sh, staging, p, bias, residual, (warp - 2) >> 2, warp & 3, lane, order, &map_c, &map_y);
  }
  __syncwarp();
  teardown(sh, warp);
}

// Largest number of co-resident clusters of two CTAs (falls back to one per two SMs).
static int max_clusters() {
  static int n = 0;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(gemm_bf16_pair_kernel<PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    cudaFuncSetAttribute(gemm_bf16_pair_kernel<WITH_GELU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    cudaFuncSetAttribute(gemm_bf16_pair_kernel<RESIDUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2 * (gemm_sm_count() / 2)); cfg.blockDim = dim3(GROUP_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES; cfg.attrs = at; cfg.numAttrs = 1;
    int c = 0;
    if (cudaOccupancyMaxActiveClusters(&c, (void*)gemm_bf16_pair_kernel<PLAIN>, &cfg) == cudaSuccess && c > 0) n = c;
    else { cudaGetLastError(); n = gemm_sm_count() / 2; }
  });
  return n;
}

// Columns of a tile.  A launch takes ceil(tiles / clusters) rounds of a tile's time, which is its columns' MMAs or, for
// narrow tiles, the operands' way out of L2: per 64-wide K block and CTA 32, 28 or 24 KB at about 64 bytes per cycle,
// against 512, 384 or 256 cycles of MMAs.  So 48 tiles of 256 on 74 clusters (3072 x 1024: one round, 26 clusters idle)
// lose to 72 tiles of 192, and 16 tiles of 256 (1024 x 1024) to 32 of 128, whose epilogue is half as long, too.
// Measured: 3072 x 1024, K = 8192: 55 -> 46 us; 1024^3: 13.9 -> 10.2 (with the epilogue of
// gemm_pair.cuh), 256 x 1000 x 2048: 14.4 -> 10.3.
static int tile_columns(int tiles_m, int N, int clusters) {
  auto cost = [&](int bn, int cycles) { return (long long)((tiles_m * (long long)((N + bn - 1) / bn) + clusters - 1) / clusters) * cycles; };
  const long long c256 = cost(256, 512), c192 = cost(192, 448), c128 = cost(128, 384);
  if (100 * c128 < 95 * std::min(c256, c192)) return 128;
  return 100 * c192 < 95 * c256 ? 192 : 256;
}

}  // namespace gemm2

// Shapes the pair kernel takes: TMA-storable C and at least one full pair tile each way.
bool gemm_pair_applicable(const void* C, int M, int N, int K, int flags) {
  const bool a_km = (flags & gemm::A_IS_KM) != 0, b_kn = (flags & gemm::B_IS_KN) != 0;
  if (M < 2 * gemm2::BM || N < gemm2::BN || N % 8 || ((uintptr_t)C & 15)) return false;
  if ((a_km ? M : K) % 8) return false;          // 16-byte rows of A as stored
  if (!b_kn && K % 8) return false;              // 16-byte rows of B as stored ([K, N] rows are covered by N % 8)
  return true;
}

// lda / ldb / ldc: row pitch of A, B, C as stored, in elements (0: dense).  With explicit pitches the
// extents themselves need not be multiples of 8 (a [T, 50257] matrix held in rows of 50264).
// gelu_out (optional): a second [M, N] matrix with C's pitch that receives gelu(C); residual (optional, not both): a dense [M, N]
// matrix that is added to C.
int launch_gemm_pair(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int epilogue,
                     int* status_word, cudaStream_t stream, int64_t lda, int64_t ldb, int64_t ldc, void* gelu_out, const void* residual) {
  CUtensorMap ma, mb, mc, my;
  int st;
  const int clusters = gemm2::max_clusters();
  const int tiles_m = (M + 2 * gemm2::BM - 1) / (2 * gemm2::BM);
  const int bn = gemm2::tile_columns(tiles_m, N, clusters);
  const bool a_km = (epilogue & gemm::A_IS_KM) != 0;       // A given as [K, M], M contiguous
  if (!lda) lda = a_km ? M : K;
  if (a_km) st = make_tmap_bf16(&ma, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, gemm2::BK);
  else st = make_tmap_bf16(&ma, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, gemm2::BM);
  if (st) return st;
  const bool b_kn = (epilogue & gemm::B_IS_KN) != 0;       // B given as [K, N], N contiguous
  if (!ldb) ldb = b_kn ? N : K;
  if (b_kn) st = make_tmap_bf16(&mb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, gemm2::BK);
  else st = make_tmap_bf16(&mb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, bn / 2);
  if (st) return st;
  if (!ldc) ldc = N;
  if ((st = make_tmap_bf16(&mc, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, gemm2::BM))) return st;
  my = mc;
  if (gelu_out && (st = make_tmap_bf16(&my, gelu_out, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, gemm2::BM))) return st;
  gemm::Problem p{};
  p.M = M; p.N = N; p.K = K;
  p.tiles_m = tiles_m;
  p.tiles_n = (N + bn - 1) / bn;
  p.pair_n = bn;
  p.k_blocks = (K + gemm2::BK - 1) / gemm2::BK;
  p.epilogue = epilogue & 3;
  p.b_mn = b_kn ? 1 : 0;
  p.a_mn = a_km ? 1 : 0;
  p.bias = (const __nv_bfloat16*)bias;
  p.residual = (const __nv_bfloat16*)residual;
  p.tma_store = 1;
  p.status = status_word;
  const int nclusters = std::min(p.tiles_m * p.tiles_n, clusters);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see pdl.cuh
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(2 * nclusters); cfg.blockDim = dim3(gemm2::GROUP_THREADS);
  cfg.dynamicSmemBytes = gemm2::SMEM_BYTES; cfg.stream = stream; cfg.attrs = at; cfg.numAttrs = 2;
  const auto kernel = gelu_out ? gemm2::gemm_bf16_pair_kernel<gemm2::WITH_GELU> : residual ? gemm2::gemm_bf16_pair_kernel<gemm2::RESIDUAL>
                                                                                           : gemm2::gemm_bf16_pair_kernel<gemm2::PLAIN>;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mb, mc, my, p);
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "pair gemm launch: %s", cudaGetErrorString(e));
}

}  // namespace tmpi
