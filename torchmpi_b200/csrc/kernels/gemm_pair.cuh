// The bf16 tcgen05 GEMM on CTA pairs (cta_group::2): two CTAs of a cluster, on the two SMs of a
// TPC, compute one 256 x 256 output tile.
//
// Each CTA stages 128 rows of A and 128 rows of B (its half of the 256 columns of the tile) per
// 64-wide K block, so a stage is 32 KB and six stages fit beside the epilogue staging.  One thread
// of the even CTA issues tcgen05.mma.cta_group::2 with M = 256, N = 256: both tensor cores read
// their own A half and both B halves, which halves the shared-memory traffic per FLOP against a
// 128 x 256 tile on one CTA.  Each CTA keeps the 128 accumulator rows of its A half in its own
// tensor memory (two 256-column accumulators) and runs its own epilogue.
//
// Synchronisation (all waits bounded, as in gemm_core.cuh):
//   full[s]   lives in the even CTA; both producers' TMA loads count their bytes there
//   empty[s]  one per CTA; the issuer commits to both after the MMAs of the stage
//   acc_full  one per CTA; the issuer commits to both after the last K block of a tile
//   acc_empty lives in the even CTA; the epilogue warps of the pair (four or eight per CTA) arrive there
// The roles take the same hooks as the single-CTA ones; m_blk counts 128-row blocks, so the hooks of
// the fused kernels (rows-ready wait, destination map) apply per CTA.
#pragma once
#include "gelu.cuh"
#include "gemm_core.cuh"

namespace tmpi {
namespace gemm2 {

using gemm::Problem;
constexpr int BM = 128;               // rows per CTA; the pair covers 2 * BM
constexpr int BN = 256;               // columns of the pair's tile; each CTA stages BN / 2 rows of B
constexpr int BK = 64, STAGES = 6, UMMA_K = 16;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = (BN / 2) * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int THREADS = 192;
constexpr int TMEM_COLS = 512;
constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_BYTES + gemm::EPI_STAGING_BYTES + 1024 + 256;
constexpr unsigned long long kWaitBudgetNs = gemm::kWaitBudgetNs;
static_assert(BN == gemm::BN && BM == gemm::BM, "the epilogue is shared with the single-CTA kernel");
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");

// Tiles are visited in bands of 8 tile-rows, so that the clusters running at one time share B panels in L2.
constexpr int BAND = 8;   // 256-row tiles per band

__device__ __forceinline__ void band_order(int t, int tiles_m, int tiles_n, int* m_tile, int* n_blk) {
  const int per_band = BAND * tiles_n;
  const int band = t / per_band;
  const int rows = min(BAND, tiles_m - band * BAND);
  const int r = t - band * per_band;
  *m_tile = band * BAND + r % rows;
  *n_blk = r / rows;
}

struct Shared {
  uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int error;
};

// NST: stages of the operand ring in use; one fewer leaves its 32 KB to the epilogue's staging.
template <int NST = STAGES>
__device__ __forceinline__ void carve(unsigned char* raw, unsigned char** tiles, Shared** sh, unsigned char** staging) {
  uintptr_t base = ((uintptr_t)raw + 1023) & ~(uintptr_t)1023;
  *tiles = (unsigned char*)base;
  *staging = (unsigned char*)(base + (size_t)NST * STAGE_BYTES);
  *sh = (Shared*)(base + (size_t)STAGES * STAGE_BYTES + gemm::EPI_STAGING_BYTES);
}

// All threads of both CTAs.  The dynamic shared memory has the same layout in both CTAs, so an
// offset taken in one is valid in the other.
__device__ __forceinline__ void setup(Shared* sh, int warp, const CUtensorMap* ma, const CUtensorMap* mb, int epilogue_warps = 4) {
  if (warp == 0 && sm100::elect_one()) {
    sm100::tma_prefetch_desc(ma);
    sm100::tma_prefetch_desc(mb);
    for (int s = 0; s < STAGES; ++s) { sm100::mbar_init(&sh->full[s], 1); sm100::mbar_init(&sh->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { sm100::mbar_init(&sh->acc_full[a], 1); sm100::mbar_init(&sh->acc_empty[a], 2 * epilogue_warps); }
    sh->error = 0;
    sm100::fence_barrier_init();
  }
  if (warp == 1) {
    sm100::tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
    sm100::tmem_relinquish_pair();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::cluster_sync();          // the other CTA's barriers exist before anything signals them
  sm100::tc_fence_after();
}

// One thread in EACH CTA.  order(it, &m_blk, &n_blk): m_blk is this CTA's 128-row block.
template <int NST = STAGES, typename TileOrder, typename ASource>
__device__ __forceinline__ void producer(Shared* sh, unsigned char* tiles, const Problem& p, const CUtensorMap* ma,
                                         const CUtensorMap* mb, uint32_t rank, TileOrder order, ASource a_source) {
  const int bn = p.pair_n ? p.pair_n : BN;
  // bytes of B per stage and CTA: bn / 2 rows, or (MN-major) whole 64-column boxes, of which bn / 2 columns are used
  const bool two_boxes = bn / 2 > 64;
  const uint32_t stage_tx = 2 * (A_BYTES + (p.b_mn ? (two_boxes ? B_BYTES : B_BYTES / 2) : (bn / 2) * BK * 2));
  int stage = 0;
  uint32_t phase = 0;
  int m_blk, n_blk;
  for (int it = 0; order(it, &m_blk, &n_blk); ++it) {
    const CUtensorMap* a_map = ma;
    int a_row0 = m_blk * BM;
    if (!a_source(m_blk, &a_map, &a_row0)) { gemm::fail(sh, p, 11); return; }
    const int b_row0 = n_blk * bn + (int)rank * (bn / 2);
    for (int kb = 0; kb < p.k_blocks; ++kb) {
      if (!sm100::mbar_wait(&sh->empty[stage], phase ^ 1, kWaitBudgetNs) || sh->error) { gemm::fail(sh, p, 12); return; }
      unsigned char* a_dst = tiles + (size_t)stage * STAGE_BYTES;
      const uint32_t full0 = sm100::map_to_cta(&sh->full[stage], 0);
      if (rank == 0) sm100::mbar_expect_tx(&sh->full[stage], stage_tx);   // both CTAs' bytes
      if (!p.a_mn) {
        sm100::tma_load_2d_pair(a_dst, a_map, kb * BK, a_row0, full0);
      } else {   // A is [K, M]: two boxes of 64 rows of the product x 64 k-rows
        sm100::tma_load_2d_pair(a_dst, a_map, a_row0, kb * BK, full0);
        sm100::tma_load_2d_pair(a_dst + A_BYTES / 2, a_map, a_row0 + 64, kb * BK, full0);
      }
      if (!p.b_mn) {
        sm100::tma_load_2d_pair(a_dst + A_BYTES, mb, kb * BK, b_row0, full0);
      } else {   // B is [K, N]: two boxes of 64 columns x 64 k-rows, each a column of eight swizzle atoms
        sm100::tma_load_2d_pair(a_dst + A_BYTES, mb, b_row0, kb * BK, full0);
        if (two_boxes) sm100::tma_load_2d_pair(a_dst + A_BYTES + B_BYTES / 2, mb, b_row0 + 64, kb * BK, full0);
      }
      if (++stage == NST) { stage = 0; phase ^= 1; }
    }
  }
}

// One thread of the EVEN CTA only.
template <int NST = STAGES, typename TileOrder>
__device__ __forceinline__ void mma_issuer(Shared* sh, unsigned char* tiles, const Problem& p, TileOrder order) {
  const uint32_t idesc = sm100::make_idesc_f16(2 * BM, p.pair_n ? p.pair_n : BN, true, p.b_mn != 0, p.a_mn != 0);
  int stage = 0;
  uint32_t phase = 0;
  int m_blk, n_blk;
  for (int it = 0; order(it, &m_blk, &n_blk); ++it) {
    const int acc = it & 1;
    const uint32_t acc_phase = (it >> 1) & 1;
    if (!sm100::mbar_wait(&sh->acc_empty[acc], acc_phase ^ 1, kWaitBudgetNs) || sh->error) { gemm::fail(sh, p, 13); return; }
    sm100::tc_fence_after();
    const uint32_t d_tmem = sh->tmem_base + (uint32_t)acc * BN;
    for (int kb = 0; kb < p.k_blocks; ++kb) {
      if (!sm100::mbar_wait(&sh->full[stage], phase, kWaitBudgetNs) || sh->error) { gemm::fail(sh, p, 14); return; }
      sm100::tc_fence_after();
      const uint32_t a_addr = sm100::smem_u32(tiles + (size_t)stage * STAGE_BYTES);
      const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) {
        const uint64_t da = p.a_mn ? sm100::make_desc_sw128_mn(a_addr + k * UMMA_K * 128, A_BYTES / 2, 1024)
                                   : sm100::make_desc_sw128(a_addr + k * UMMA_K * 2);
        const uint64_t db = p.b_mn ? sm100::make_desc_sw128_mn(b_addr + k * UMMA_K * 128, B_BYTES / 2, 1024)
                                   : sm100::make_desc_sw128(b_addr + k * UMMA_K * 2);
        sm100::umma_f16_pair(d_tmem, da, db, idesc, (kb | k) != 0);
      }
      sm100::umma_commit_pair(sm100::map_to_cta(&sh->empty[stage], 0));   // both producers may refill the stage
      sm100::umma_commit_pair(sm100::map_to_cta(&sh->empty[stage], 1));
      if (++stage == NST) { stage = 0; phase ^= 1; }
    }
    sm100::umma_commit_pair(sm100::map_to_cta(&sh->acc_full[acc], 0));    // both epilogues may read
    sm100::umma_commit_pair(sm100::map_to_cta(&sh->acc_full[acc], 1));
  }
}

// The four epilogue warps of EACH CTA (see gemm::epilogue_tma_impl for DestMap; leaving the map
// null skips the stores of a row block).
template <typename TileOrder, typename DestMap>
__device__ __forceinline__ void epilogue(Shared* sh, unsigned char* staging, const Problem& p, int quarter, int lane,
                                         TileOrder order, DestMap dest) {
  gemm::epilogue_tma_impl(sh, staging, p, quarter, lane, order, dest, [sh](int acc) {
    sm100::mbar_arrive_cluster(sm100::map_to_cta(&sh->acc_empty[acc], 0));
  });
}

// The epilogue of the plain GEMM: two groups of four warps in EACH CTA take the 64-column slices of a tile in turn, each
// through a staging tile of its own, so that one group converts while the other waits for its accumulator reads and its
// staging tile.  With one group the four slices of a tile were a serial chain of about 1 us each that a product with a
// short K (16 K blocks: 4.3 us of MMAs per tile) could not hide, and that every launch paid at its end.  The bias of a
// slice is read as eight 16-byte loads (64 scalar loads before).  Measured, 8192 x 4096 x 1024 with a bias: 83 -> 52 us; without
// one 59 -> 50; 8192 x 50264 x 1024: 694 -> 585; 1024^3, where the launch is one tile and its epilogue: 17 -> 15.
// TWO: gelu(C) is written beside C (map2): GELU of the rounded bf16 value, which is what a separate pass over C computes,
// without that pass's launch and its read of C.  It has staging tiles of its own (the operand ring gives up a stage for
// them), so a group never waits for the store it has just issued.  8192 x 4096 x 1024: product 83 and pass 36 us before, one
// kernel of 69 now (82 with one staging tile per group).
// RESIDUAL: the residual is added before the rounding.  A thread reads its row's 128 bytes of the next slice while it works on this one.
// (A pass that adds after the product reads both and writes the sum: 8 us at 8192 x 1024.)
enum { PLAIN = 0, WITH_GELU = 1, RESIDUAL = 2 };
constexpr int GROUPS = 2, GROUP_THREADS = 64 + GROUPS * 128;

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

template <int MODE, typename TileOrder>
__device__ __forceinline__ void epilogue_groups(Shared* sh, unsigned char* staging, const Problem& p, const __nv_bfloat16* bias,
                                                const __nv_bfloat16* residual, int group, int quarter, int lane, TileOrder order, const CUtensorMap* map_c, const CUtensorMap* map2) {
  constexpr bool TWO = MODE == WITH_GELU;
  constexpr int SLICE = 64, SLICE_BYTES = BM * SLICE * 2;
  static_assert(GROUPS * SLICE_BYTES <= gemm::EPI_STAGING_BYTES && GROUPS * SLICE_BYTES <= STAGE_BYTES, "a staging tile per group and output");
  const int row = quarter * 32 + lane;
  const bool leader = quarter == 0 && lane == 0;
  const int bn = p.pair_n ? p.pair_n : BN;
  unsigned char* stg0 = staging + group * SLICE_BYTES;
  const bool bias_vec = ((uintptr_t)bias & 15) == 0;
  int m_blk, n_blk;
  uint4 res[8], res_next[8];
  auto read_residual = [&](uint4 (&v)[8], int col0) {
    const long long at = (long long)(m_blk * BM + row) * p.N + col0;
    const bool inside = m_blk * BM + row < p.M;
#pragma unroll
    for (int j = 0; j < 8; ++j)          // N is a multiple of 8
      v[j] = inside && col0 + 8 * j < p.N ? __ldg(reinterpret_cast<const uint4*>(residual + at) + j) : make_uint4(0u, 0u, 0u, 0u);
  };
  for (int it = 0; order(it, &m_blk, &n_blk); ++it) {
    const int acc = it & 1;
    if (MODE == RESIDUAL) read_residual(res_next, n_blk * bn + group * SLICE);
    const uint32_t ok = sm100::mbar_wait(&sh->acc_full[acc], (it >> 1) & 1, kWaitBudgetNs) && !sh->error;
    uint32_t all_ok;                    // the group meets at named barriers below: it goes on, or leaves, together
    asm volatile("{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n barrier.cta.red.and.pred q, %2, 128, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(all_ok) : "r"(ok), "r"(1 + group) : "memory");
    if (!all_ok) { gemm::fail(sh, p, 5); break; }
    sm100::tc_fence_after();
    const int row0 = m_blk * BM;
    const bool store = leader && row0 < p.M;
    const uint32_t t_base = sh->tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * BN;
#pragma unroll 1
    for (int c0 = group * SLICE; c0 < bn; c0 += GROUPS * SLICE) {
      const int col0 = n_blk * bn + c0;
      if (col0 >= p.N) break;           // uniform over the group: the rest of the tile lies outside C
      uint32_t r[2][32], w[32];
      sm100::tmem_ld_32x32(t_base + c0, r[0]);
      sm100::tmem_ld_32x32(t_base + c0 + 32, r[1]);
      if (MODE == RESIDUAL) {
#pragma unroll
        for (int j = 0; j < 8; ++j) res[j] = res_next[j];
        if (c0 + GROUPS * SLICE < bn) read_residual(res_next, col0 + GROUPS * SLICE);
      }
      sm100::tmem_ld_wait();
      if (p.epilogue & gemm::EPI_BIAS) {
        if (bias_vec && col0 + SLICE <= p.N) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(bias + col0) + j);
            const uint32_t b[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t* v = &r[j >> 2][(j & 3) * 8 + 2 * q];
              v[0] = __float_as_uint(__uint_as_float(v[0]) + __uint_as_float(b[q] << 16));
              v[1] = __float_as_uint(__uint_as_float(v[1]) + __uint_as_float(b[q] & 0xffff0000u));
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (col0 + j < p.N) r[j >> 5][j & 31] = __float_as_uint(__uint_as_float(r[j >> 5][j & 31]) + __bfloat162float(bias[col0 + j]));
        }
      }
      if (MODE == RESIDUAL) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t b[4] = {res[j].x, res[j].y, res[j].z, res[j].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t* v = &r[j >> 2][(j & 3) * 8 + 2 * q];
            v[0] = __float_as_uint(__uint_as_float(v[0]) + __uint_as_float(b[q] << 16));
            v[1] = __float_as_uint(__uint_as_float(v[1]) + __uint_as_float(b[q] & 0xffff0000u));
          }
        }
      }
      if (p.epilogue & gemm::EPI_GELU) {
#pragma unroll
        for (int j = 0; j < 64; ++j) r[j >> 5][j & 31] = __float_as_uint(gemm::gelu_erf(__uint_as_float(r[j >> 5][j & 31])));
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[j >> 4][2 * (j & 15)]), __uint_as_float(r[j >> 4][2 * (j & 15) + 1]));
        w[j] = *reinterpret_cast<uint32_t*>(&h);
      }
      auto put = [&](const CUtensorMap* map, int which) {
        unsigned char* stg = stg0 + which * GROUPS * SLICE_BYTES;
        unsigned char* stg_row = stg + row * 128;
        // the store that used this staging tile before must have read it (TWO: the other tile's may still be at it)
        if (leader) {
          if (TWO) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        group_sync(group);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          *reinterpret_cast<uint4*>(stg_row + ((u ^ (row & 7)) << 4)) = make_uint4(w[4 * u], w[4 * u + 1], w[4 * u + 2], w[4 * u + 3]);
        sm100::fence_proxy_async_smem();       // generic-proxy writes to shared memory -> visible to the TMA unit
        group_sync(group);
        if (store) sm100::tma_store_2d(map, stg, col0, row0);
        if (leader) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      };
      put(map_c, 0);
      if (TWO) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {         // bf16 -> fp32 is a shift or a mask
          float y0, y1;
          gelu_value2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u), &y0, &y1);
          __nv_bfloat162 h = __floats2bfloat162_rn(y0, y1);
          w[j] = *reinterpret_cast<uint32_t*>(&h);
        }
        put(map2, 1);
      }
    }
    sm100::tc_fence_before();
    __syncwarp();
    if (lane == 0) sm100::mbar_arrive_cluster(sm100::map_to_cta(&sh->acc_empty[acc], 0));
  }
  if (leader) {
    // the tiles have been read before the CTA gives its shared memory back; the writes themselves complete with the kernel
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
}

// All threads of both CTAs.  Neither CTA frees its tensor memory or exits while the other may still
// signal its barriers or have the pair's MMAs read its shared memory.
__device__ __forceinline__ void teardown(Shared* sh, int warp) {
  sm100::tc_fence_before();
  __syncthreads();
  if (sh->error && warp == 0 && sm100::elect_one()) {
    const unsigned long long t0 = sm100::now_ns();
    while (sm100::now_ns() - t0 < 200000000ull) { __nanosleep(1000); }   // copies in flight complete within microseconds
  }
  __syncthreads();
  sm100::cluster_sync();
  if (warp == 1) {
    sm100::tc_fence_after();
    sm100::tmem_dealloc_pair(sh->tmem_base, TMEM_COLS);
  }
}

}  // namespace gemm2
}  // namespace tmpi
