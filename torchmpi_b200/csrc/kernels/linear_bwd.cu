// The gradients of a linear layer, dX = dY W, dW = dY^T X and db = column sums of dY, in one launch on CTA pairs
// (gemm_pair.cuh): dY [rows, out], W [out, in] and X [rows, in] are read as they lie.
//
// Work units.  Each product is cut into tiles of 256 rows x bn columns, and a tile whose K is long beside what the other clusters
// have to do into slices of K.  The units of both products form one list, longest first, dealt to the persistent clusters in
// turn.  Two launches of their own each end in a partly filled round (8192 x 1024 x 1024: 128 tiles of dX on 74 clusters, then 16
// long ones of dW); in one list the short units fill what the long ones leave.
//
// A sliced tile's partial sums go to the workspace in fp32; the CTA that arrives last at its tile adds all slices in their
// order (bit-reproducible, nobody waits) and writes the result.  The arrival counters wrap to zero by themselves.
//
// db is summed by the epilogue warps, in fp32 and in short chains, before their first tile, while the MMAs of that tile run:
// units of 256 columns and a slice of the rows, dealt from the last cluster on, which has the fewest tiles.  (As a product,
// dY^T times a column of ones, it was one chain of rows / 16 steps, in which small values beside large ones were lost: 2046 times 2^-14
// between two values of 2^15 that cancel gave 0.  As units of the list, behind the tiles, 8192 x 1024 x 4096 took 7 us longer.)  A
// pass over dY of its own took two launches.
//
// What bounds it: the tensor cores at the clock that the power limit leaves (8192 rows), the length of one unit and the partial tiles'
// way through L2 (1024 rows and less).  Measured, captured calls in a row, rows x inputs x outputs, us, the launches that it replaces (two
// for the bias sums, one for dX, one or two for dW) and this: 64 x 512 x 512 14.5, 5.8; 256 x 2048 x 1000 21.4, 9.0; 1024 x 1024 x 1024
// 22.4, 8.8; 4096 x 512 x 512 41.7, 13.5; 8192 x 768 x 768 61.4, 25.1; 8192 x 1024 x 1024 52.7, 30.5; 8192 x 1024 x 3072 88.9, 78.5;
// 8192 x 1024 x 4096 109, 98.  With the kind of product as a run-time value in the producer's and the issuer's loops, 13 % longer.
#include "attn_util.cuh"
#include "gemm_pair.cuh"
#include "pdl.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"
#include <algorithm>
#include <mutex>

namespace tmpi {

int make_tmap_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
int gemm_sm_count();
int* gemm_status_word();

namespace lbwd {

using namespace gemm2;
enum { DX = 0, DW = 1, DB = 2 };
constexpr int EPI_THREADS = GROUPS * 128;
constexpr int DB_GROUPS = EPI_THREADS / (BM / 8);    // db: threads that share eight columns

struct Part {
  int what;
  int M, N;                  // extents of the result
  int tiles_m, tiles_n, bn;  // 256-row tiles, tiles of bn columns
  int k_blocks, per, slices; // 64-wide blocks of K, those of one slice
  int first;                 // its first unit in the list
  int arrivals;              // its first arrival counter (two per tile)
  long long ws;              // its first float of the workspace
};

struct Problem {
  Part part[2];              // the products
  Part sums;                 // db, where it is wanted (tiles_m > 0)
  int parts, total;          // total: units of the products
  float* ws;
  unsigned* arrivals;
  const __nv_bfloat16* dy;
  long long ld_dy;
  int rows, out;
  __nv_bfloat16* db;
  int* status;
};

struct Unit { int m_blk, n_blk, kb0, kb1, tile, slice; };

// f(part, unit, number of the unit in this cluster's list) for each unit of this cluster until it returns false; m_blk counts
// 128-row blocks (of this CTA).
template <typename F>
__device__ __forceinline__ void for_units(const Problem& p, uint32_t rank, F f) {
  const int step = (int)(gridDim.x >> 1);
  int at = (int)(blockIdx.x >> 1), it = 0;
  for (int i = 0; i < p.parts; ++i) {
    const Part& q = p.part[i];
    const int tiles = q.tiles_m * q.tiles_n, end = q.first + tiles * q.slices;
    for (; at < end; at += step, ++it) {
      Unit u;
      const int r = at - q.first;
      u.slice = r / tiles;             // the tiles of one slice run together and share its operands in L2
      u.tile = r - u.slice * tiles;
      int m_tile;
      band_order(u.tile, q.tiles_m, q.tiles_n, &m_tile, &u.n_blk);
      u.m_blk = m_tile * 2 + (int)rank;
      u.kb0 = u.slice * q.per;
      u.kb1 = min(q.k_blocks, u.kb0 + q.per);
      if (!f(q, u, it)) return;
    }
  }
}

struct Sh { Shared s; int last; };
static_assert(sizeof(Sh) <= 256, "barriers");

__device__ __forceinline__ void give_up(Shared* sh, const Problem& p, int where) {
  atomicExch(&sh->error, where);
  if (p.status) atomicCAS(p.status, 0, 1000 + where);
}

struct Ring { int stage; uint32_t phase; };
__device__ __forceinline__ void advance(Ring* r) { if (++r->stage == STAGES) { r->stage = 0; r->phase ^= 1; } }

// One thread in each CTA.
template <int WHAT>
__device__ __forceinline__ bool produce_unit(Shared* sh, unsigned char* tiles, const Problem& p, const CUtensorMap* ma, const CUtensorMap* mb,
                                             uint32_t rank, int bn, const Unit& u, Ring* ring) {
  const int half = bn / 2, m0 = u.m_blk * BM, n0 = u.n_blk * bn + (int)rank * half;
  const bool two = half > 64;
  // bytes of a stage in both CTAs: A, and one or two boxes of 64 columns of B, of which bn / 2 columns are used
  const uint32_t tx = 2 * (A_BYTES + (two ? B_BYTES : B_BYTES / 2));
  for (int kb = u.kb0; kb < u.kb1; ++kb) {
    const int stage = ring->stage;
    if (!sm100::mbar_wait(&sh->empty[stage], ring->phase ^ 1, kWaitBudgetNs) || sh->error) { give_up(sh, p, 21); return false; }
    unsigned char* dst = tiles + (size_t)stage * STAGE_BYTES;
    const uint32_t full0 = sm100::map_to_cta(&sh->full[stage], 0);
    if (rank == 0) sm100::mbar_expect_tx(&sh->full[stage], tx);
    const int k0 = kb * BK;
    if (WHAT == DX) {          // rows of dY: K contiguous
      sm100::tma_load_2d_pair(dst, ma, k0, m0, full0);
      sm100::tma_load_2d_pair(dst + A_BYTES / 2, ma, k0, m0 + 64, full0);
    } else {                   // columns of dY: M contiguous
      sm100::tma_load_2d_pair(dst, ma, m0, k0, full0);
      sm100::tma_load_2d_pair(dst + A_BYTES / 2, ma, m0 + 64, k0, full0);
    }
    sm100::tma_load_2d_pair(dst + A_BYTES, mb, n0, k0, full0);
    if (two) sm100::tma_load_2d_pair(dst + A_BYTES + B_BYTES / 2, mb, n0 + 64, k0, full0);
    advance(ring);
  }
  return true;
}

// One thread of the even CTA.
template <int WHAT>
__device__ __forceinline__ bool issue_unit(Shared* sh, unsigned char* tiles, const Problem& p, int bn, const Unit& u, int it, Ring* ring) {
  const uint32_t idesc = sm100::make_idesc_f16(2 * BM, bn, true, true, WHAT == DW);
  const int acc = it & 1;
  if (!sm100::mbar_wait(&sh->acc_empty[acc], ((it >> 1) & 1) ^ 1, kWaitBudgetNs) || sh->error) { give_up(sh, p, 22); return false; }
  sm100::tc_fence_after();
  const uint32_t d = sh->tmem_base + (uint32_t)acc * BN;
  for (int kb = u.kb0; kb < u.kb1; ++kb) {
    const int stage = ring->stage;
    if (!sm100::mbar_wait(&sh->full[stage], ring->phase, kWaitBudgetNs) || sh->error) { give_up(sh, p, 23); return false; }
    sm100::tc_fence_after();
    const uint32_t a = sm100::smem_u32(tiles + (size_t)stage * STAGE_BYTES), b = a + A_BYTES;
#pragma unroll
    for (int k = 0; k < BK / UMMA_K; ++k) {
      const uint64_t da = WHAT == DX ? sm100::make_desc_sw128(a + k * UMMA_K * 2) : sm100::make_desc_sw128_mn(a + k * UMMA_K * 128, A_BYTES / 2, 1024);
      const uint64_t db = sm100::make_desc_sw128_mn(b + k * UMMA_K * 128, B_BYTES / 2, 1024);
      sm100::umma_f16_pair(d, da, db, idesc, (uint32_t)(kb > u.kb0) | (uint32_t)k);
    }
    sm100::umma_commit_pair(sm100::map_to_cta(&sh->empty[stage], 0));
    sm100::umma_commit_pair(sm100::map_to_cta(&sh->empty[stage], 1));
    advance(ring);
  }
  sm100::umma_commit_pair(sm100::map_to_cta(&sh->acc_full[acc], 0));
  sm100::umma_commit_pair(sm100::map_to_cta(&sh->acc_full[acc], 1));
  return true;
}

__device__ __forceinline__ void all_sync() { asm volatile("bar.sync 3, %0;" ::"n"(EPI_THREADS) : "memory"); }

// The sums of 128 columns of dY from col0 over the rows [r0, r1), by all epilogue threads; thread `row` of group 0 has column col0 + row.
// Sixteen threads share eight columns, each with 16-byte loads of every 16th row, of which 8 to 16 are in flight; the values of two batches
// of eight are added as a tree, and so are the threads' sums: a value passes 8 additions and one per 256 rows.  part: 8 KB of group 0's staging.
__device__ __forceinline__ float column_sums(const Problem& p, const __nv_bfloat16* dy, float* part, int col0, int r0, int r1, int group, int row) {
  constexpr int U = 8, STEP = DB_GROUPS;
  const int e = threadIdx.x - 64, col = col0 + (e % (BM / 8)) * 8, mine = e / (BM / 8);
  const bool whole = col + 8 <= p.out;
  // a last row may end with its last column; its part of an incomplete group of columns is read one by one
  const int end = col >= p.out ? r0 : whole ? r1 : min(r1, p.rows - 1);
  unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};                      // two columns each
  auto load = [&](uint4 (&v)[U], unsigned r) {
#pragma unroll
    for (int i = 0; i < U; ++i)
      v[i] = r + i * STEP < (unsigned)end ? __ldcg(reinterpret_cast<const uint4*>(dy + (r + i * STEP) * p.ld_dy + col)) : make_uint4(0u, 0u, 0u, 0u);
  };
  auto sum = [&](const uint4 (&v)[U], unsigned long long (&to)[4]) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      unsigned long long t[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const uint32_t b = w == 0 ? v[i].x : w == 1 ? v[i].y : w == 2 ? v[i].z : v[i].w;
        t[i] = attn_util::pack2(b << 16, b & 0xffff0000u);
      }
#pragma unroll
      for (int n = U / 2; n; n /= 2)
#pragma unroll
        for (int i = 0; i < n; ++i) t[i] = attn_util::add2(t[i], t[i + n]);
      to[w] = t[0];
    }
  };
  uint4 a[U], b[U];
  load(a, r0 + mine);
  for (unsigned r = r0 + mine; r < (unsigned)end; r += 2 * U * STEP) {
    unsigned long long first[4], second[4];
    load(b, r + U * STEP);
    sum(a, first);
    load(a, r + 2 * U * STEP);
    sum(b, second);
#pragma unroll
    for (int w = 0; w < 4; ++w) acc[w] = attn_util::add2(acc[w], attn_util::add2(first[w], second[w]));
  }
  float s[8];
#pragma unroll
  for (int w = 0; w < 4; ++w) attn_util::unpack2(acc[w], s[2 * w], s[2 * w + 1]);
  if (!whole && r1 == p.rows && (r1 - 1 - r0) % STEP == mine)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (col + k < p.out) s[k] += __bfloat162float(dy[(r1 - 1) * p.ld_dy + col + k]);
  all_sync();                          // the sums of the unit before have been read
  float4* to = reinterpret_cast<float4*>(part + e * 8);
  to[0] = make_float4(s[0], s[1], s[2], s[3]);
  to[1] = make_float4(s[4], s[5], s[6], s[7]);
  all_sync();
  if (group) return 0.f;
  float t[DB_GROUPS];
#pragma unroll
  for (int g = 0; g < DB_GROUPS; ++g) t[g] = part[g * BM + row];
#pragma unroll
  for (int n = DB_GROUPS / 2; n; n /= 2)
#pragma unroll
    for (int g = 0; g < n; ++g) t[g] += t[g + n];
  return t[0];
}

// The eight epilogue warps of each CTA: two groups of four, which take the 64-column slices of a tile in turn.
__device__ __forceinline__ void finish(Sh* shl, unsigned char* staging, const Problem& p, const CUtensorMap* mdx, const CUtensorMap* mdw,
                                       const __nv_bfloat16* dy, uint32_t rank, int group, int quarter, int lane) {
  Shared* sh = &shl->s;
  constexpr int SLICE = 64, SLICE_BYTES = BM * SLICE * 2;
  const int row = quarter * 32 + lane;
  const bool leader = quarter == 0 && lane == 0;
  unsigned char* stg = staging + group * SLICE_BYTES;
  unsigned char* stg_row = stg + row * 128;
  // Whether this CTA is the last of a tile's S slices; their partial sums are then visible to all its epilogue threads.
  auto arrive = [&](const Part& q, int tile) -> bool {
    __threadfence();
    all_sync();
    const unsigned S = (unsigned)q.slices;
    if (group == 0 && leader) shl->last = atomicInc(&p.arrivals[q.arrivals + 2 * tile + (int)rank], S - 1) == S - 1;
    all_sync();
    const bool last = shl->last != 0;
    if (last) __threadfence();
    return last;
  };
  if (p.sums.tiles_m) {
    const Part& q = p.sums;
    const int S = q.slices, clusters = (int)(gridDim.x >> 1);
    for (int at = clusters - 1 - (int)(blockIdx.x >> 1); at < q.tiles_m * S; at += clusters) {
      const int slice = at / q.tiles_m, tile = at - slice * q.tiles_m, col0 = (2 * tile + (int)rank) * BM;
      const int r0 = slice * q.per * BK, r1 = (int)min((long long)(slice + 1) * q.per * BK, (long long)p.rows);
      float sum = column_sums(p, dy, reinterpret_cast<float*>(staging), col0, r0, r1, group, row);
      bool write = true;
      if (S > 1) {
        float* ws = p.ws + q.ws + ((long long)tile * S * 2 + (int)rank) * BM + row;      // of slice 0; the next one 2 * BM further
        if (group == 0) __stcg(ws + 2LL * BM * slice, sum);
        write = arrive(q, tile);
        if (write && group == 0) {
          sum = 0.f;
          for (int s = 0; s < S; s += 4) {
            float t[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = s + k < S ? __ldcg(ws + 2LL * BM * (s + k)) : 0.f;
            sum += (t[0] + t[1]) + (t[2] + t[3]);
          }
        }
      }
      if (write && group == 0 && col0 + row < p.out) p.db[col0 + row] = __float2bfloat16_rn(sum);
    }
  }
  for_units(p, rank, [&](const Part& q, const Unit& u, int it) -> bool {
    const int S = q.slices, M = q.M, row0 = u.m_blk * BM;
    // slot of a slice: 128 rows x bn columns as [column / 4][row][4]
    const long long slot = (long long)q.bn * BM;
    float* ws = p.ws + q.ws + ((long long)u.tile * S * 2 + (int)rank) * slot;      // of slice 0; the next one 2 * slot further
    const int acc = it & 1, N = q.N, bn = q.bn;
    const uint32_t ok = sm100::mbar_wait(&sh->acc_full[acc], (it >> 1) & 1, kWaitBudgetNs) && !sh->error;
    uint32_t all_ok;                    // the warps meet below: they go on, or leave, together
    asm volatile("{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n barrier.cta.red.and.pred q, 3, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(all_ok) : "r"(ok), "n"(EPI_THREADS) : "memory");
    if (!all_ok) { give_up(sh, p, 24); return false; }
    sm100::tc_fence_after();
    const uint32_t t_base = sh->tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * BN;
    auto release = [&] {                // the accumulator has been read
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive_cluster(sm100::map_to_cta(&sh->acc_empty[acc], 0));
    };
    const CUtensorMap* map = q.what == DX ? mdx : mdw;
    auto put = [&](const uint32_t (&r)[2][32], int col0) {
      if (leader) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      group_sync(group);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 8 * j + 2 * e;
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[c >> 5][c & 31]), __uint_as_float(r[c >> 5][(c & 31) + 1]));
          w[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(stg_row + ((j ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      sm100::fence_proxy_async_smem();
      group_sync(group);
      if (leader) {
        if (row0 < M) sm100::tma_store_2d(map, stg, col0, row0);
        if (row0 + 64 < M) sm100::tma_store_2d(map, stg + SLICE_BYTES / 2, col0, row0 + 64);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    };
#pragma unroll 1
    for (int c0 = group * SLICE; c0 < bn && u.n_blk * bn + c0 < N; c0 += GROUPS * SLICE) {
      uint32_t r[2][32];
      sm100::tmem_ld_32x32(t_base + c0, r[0]);
      sm100::tmem_ld_32x32(t_base + c0 + 32, r[1]);
      sm100::tmem_ld_wait();
      if (S == 1) {
        put(r, u.n_blk * bn + c0);
      } else {
        float4* to = reinterpret_cast<float4*>(ws + 2 * slot * u.slice) + (c0 / 4) * BM + row;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t* v = &r[j >> 3][(j & 7) * 4];
          __stcg(to + j * BM, make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]), __uint_as_float(v[3])));
        }
      }
    }
    release();
    if (S > 1 && arrive(q, u.tile)) {
#pragma unroll 1
      for (int c0 = group * SLICE; c0 < bn && u.n_blk * bn + c0 < N; c0 += GROUPS * SLICE) {
        uint32_t r[2][32];
#pragma unroll
        for (int j = 0; j < 64; ++j) r[j >> 5][j & 31] = 0u;
#pragma unroll 1
        for (int s = 0; s < S; ++s) {
          const float4* from = reinterpret_cast<const float4*>(ws + 2 * slot * s) + (c0 / 4) * BM + row;
          float4 v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __ldcg(from + j * BM);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            uint32_t* a = &r[j >> 3][(j & 7) * 4];
            a[0] = __float_as_uint(__uint_as_float(a[0]) + v[j].x);
            a[1] = __float_as_uint(__uint_as_float(a[1]) + v[j].y);
            a[2] = __float_as_uint(__uint_as_float(a[2]) + v[j].z);
            a[3] = __float_as_uint(__uint_as_float(a[3]) + v[j].w);
          }
        }
        put(r, u.n_blk * bn + c0);
      }
    }
    return true;
  });
  if (leader) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

__global__ void __launch_bounds__(GROUP_THREADS, 1)
linear_bwd_kernel(const __grid_constant__ CUtensorMap map_dy, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                  const __grid_constant__ CUtensorMap map_dx, const __grid_constant__ CUtensorMap map_dw, const __grid_constant__ Problem p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *tiles, *staging;
  Shared* sh;
  carve(smem_raw, &tiles, &sh, &staging);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = sm100::cluster_ctarank();
  setup(sh, warp, &map_dy, &map_x, 4 * GROUPS);
  const __nv_bfloat16* dy = p.dy;
  wait_previous(dy);
  if (warp == 0) {
    if (sm100::elect_one()) {
      Ring ring{0, 0};
      for_units(p, rank, [&](const Part& q, const Unit& u, int) -> bool {
        if (q.what == DX) return produce_unit<DX>(sh, tiles, p, &map_dy, &map_w, rank, q.bn, u, &ring);
        return produce_unit<DW>(sh, tiles, p, &map_dy, &map_x, rank, q.bn, u, &ring);
      });
    }
  } else if (warp == 1) {
    if (rank == 0 && sm100::elect_one()) {
      Ring ring{0, 0};
      for_units(p, 0, [&](const Part& q, const Unit& u, int it) -> bool {
        if (q.what == DX) return issue_unit<DX>(sh, tiles, p, q.bn, u, it, &ring);
        return issue_unit<DW>(sh, tiles, p, q.bn, u, it, &ring);
      });
    }
  } else {
    finish((Sh*)sh, staging, p, &map_dx, &map_dw, dy, rank, (warp - 2) >> 2, warp & 3, lane);
  }
  __syncwarp();
  teardown(sh, warp);
}

static int max_clusters() {
  static int n = 0;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(linear_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2 * (gemm_sm_count() / 2)); cfg.blockDim = dim3(GROUP_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES; cfg.attrs = at; cfg.numAttrs = 1;
    int c = 0;
    if (cudaOccupancyMaxActiveClusters(&c, (void*)linear_bwd_kernel, &cfg) == cudaSuccess && c > 0) n = c;
    else { cudaGetLastError(); n = gemm_sm_count() / 2; }
  });
  return n;
}

// ---------------------------------------------------------------- the work list
struct Choice { int bn, slices; };
constexpr int LAUNCH_CYCLES = 14000;          // what a second launch costs, the first one's tail and the second one's first loads

static void set_part(Part* q, int what, int rows, int in, int out, Choice c) {
  q->what = what;
  q->M = what == DX ? rows : out;
  q->N = what == DB ? 1 : in;
  q->bn = what == DB ? BN : c.bn;
  q->tiles_m = (q->M + 2 * BM - 1) / (2 * BM);
  q->tiles_n = what == DB ? 1 : (in + c.bn - 1) / c.bn;
  q->k_blocks = ((what == DX ? out : rows) + BK - 1) / BK;
  q->per = (q->k_blocks + c.slices - 1) / c.slices;
  q->slices = (q->k_blocks + q->per - 1) / q->per;
}

// Cycles of a unit: those of its K blocks (the MMAs of 256 columns, the operands' way out of L2 for fewer) and its epilogue's
// share, with the partial tile's way to the workspace and back where there are slices.  Fitted to 41 shapes (8 - 8192 rows, 128 - 4096
// inputs and outputs) in up to 1500 forms each: the form that these numbers choose takes 0.7 % longer than the best of them on
// average, 7 % at most.
static int unit_cycles(const Part& q) {
  return std::min(q.per, 1 << 21) * (q.bn == 256 ? 512 : q.bn == 192 ? 403 : 342) + (q.slices > 1 ? 53 * q.bn + 11 * q.bn * q.slices / 2 : 35 * q.bn / 2);
}

struct Candidate { Choice c; int cycles, units; };

static int candidates(int what, int rows, int in, int out, int clusters, Candidate* list) {
  int n = 0;
  for (int bn = 256; bn >= 128; bn -= 64)
    for (int s : {1, 2, 3, 4, 6, 8}) {
      Part q;
      set_part(&q, what, rows, in, out, {bn, s});
      const int units = q.tiles_m * q.tiles_n * q.slices;
      // slices of eight K blocks or more, and of an output that leaves clusters idle or deals out badly; long slices (the K of a
      // vocabulary) also of more tiles: both gradients of a head of 1600 x 4096 x 32000 606 us with dX whole, 590 in three slices
      if (s == 1 || (q.slices == s && q.per >= 8 && units <= (q.per >= 32 ? 8 : 4) * clusters)) list[n++] = {{bn, s}, unit_cycles(q), units};
    }
  return n;
}

// The time of the first cluster, which has the longest unit of every round.
static long long span(const Candidate* const (&c)[2], int parts, int clusters) {
  const Candidate* o[2];
  for (int i = 0; i < parts; ++i) {          // longest first
    int j = i;
    for (; j > 0 && o[j - 1]->cycles < c[i]->cycles; --j) o[j] = o[j - 1];
    o[j] = c[i];
  }
  long long t = 0, at = 0, end = 0;
  for (int i = 0; i < parts; ++i) {
    end += o[i]->units;
    if (at < end) {
      const long long rounds = (end - at + clusters - 1) / clusters;
      t += rounds * o[i]->cycles;
      at += rounds * clusters;
    }
  }
  return t;
}

// Slices of the rows for db beside a list of `units` that takes `time`, whose longest unit takes `longest` and whose tiles of dW have
// `dw_slices`; and what db adds to that time.
// Clusters that the list leaves idle sum it for nothing, if they are enough (at 430 cycles a K block of 256 columns: 330 on an idle chip, 650 beside
// products that are bound by their loads).  Otherwise the epilogues of some of the others sum it under their first tile,
// in a multiple of dW's slices, which then bring the same rows into L2.  In a list of one round all wait for those units, above all
// where they are slices, so there every cluster takes a part.  A thread adds 24 times in the longest slice, of 96 K blocks (of
// very many rows, an eighth of them); up to 1024 rows are one slice, whose call needs no arrival counters (a microsecond of the host).
// us without db and with 1, 2, 4, 8, 16 slices: 1024 x 1024 x 1024 8.6, 8.7, 8.7, 9.2; 8192 x 1024 x 1024 30.3, 36.6, 29.9, 30.0, 30.5, 30.6;
// of that dW and db alone (64 units) 20.5, 27.7, 20.5, 22.3, 21.8, 21.5; 8192 x 1024 x 4096 95.5, 97.1, 97.3, 97.7, 98.7, 98.7; 65536 x 512 x 512
// (eight slices of dW) 80, 308, 179, 104, 80, 86, with nine 95; dW and db of 16384 x 1024 x 1024 (72 units, three slices) 35.9 and with 3, 6, 18 39.9, 37.8,
// 37.5.
static int sums_slices(int rows, int out, int units, long long time, int longest, int dw_slices, int clusters, int* added) {
  const int tiles = (out + 2 * BM - 1) / (2 * BM), k_blocks = (rows + BK - 1) / BK;
  auto slices = [&](long long per) { return (int)std::min(32LL, (k_blocks - 1) / std::max(16LL, std::min((long long)std::max(96, k_blocks / 8), per)) + 1); };
  *added = 0;
  int s = slices(longest / 430);
  if (units < clusters) {
    const int idle = slices((time - 1500) / 430);
    if (tiles * idle <= clusters - units) return idle;
    *added = dw_slices > 1 ? 3500 : 500;
    if (dw_slices > 1) s = std::max(s, std::min({32, clusters / tiles, k_blocks / 4}) / dw_slices * dw_slices);
  }
  const int whole = (s + dw_slices - 1) / dw_slices * dw_slices;
  return whole <= 32 && whole * 4 <= k_blocks ? whole : s;
}

struct Plan { Choice c[3]; bool apart; };      // apart: dX in a launch of its own, before the one of dW and db

// The best tiles and slices of the products in `want` as one list, and that list's time.
static long long best_list(int rows, int in, int out, int want, int clusters, Choice* best) {
  Candidate x[18], w[18];
  const int nx = want >> DX & 1 ? candidates(DX, rows, in, out, clusters, x) : 0, nw = want >> DW & 1 ? candidates(DW, rows, in, out, clusters, w) : 0;
  long long least = -1;
  for (int i = 0; i < std::max(1, nx); ++i)
    for (int j = 0; j < std::max(1, nw); ++j) {
      const Candidate* c[2] = {};
      int parts = 0;
      if (nx) c[parts++] = &x[i];
      if (nw) c[parts++] = &w[j];
      long long t = span(c, parts, clusters);
      int slices = 1, added = 0;
      if (want >> DB & 1) {
        int units = 0, longest = 0;
        for (int k = 0; k < parts; ++k) { units += c[k]->units; longest = std::max(longest, c[k]->cycles); }
        slices = sums_slices(rows, out, units, t, longest, nw ? w[j].c.slices : 1, clusters, &added);
        t += added;
      }
      if (least < 0 || t < least) {
        least = t;
        if (nx) best[DX] = x[i].c;
        if (nw) best[DW] = w[j].c;
        if (want >> DB & 1) best[DB] = {BN, slices};
      }
    }
  return least;
}

// The plan of a call; kept per thread for the sizes last asked for (1 - 10 us to find).
// One list has to be a twentieth shorter than two, for units of both products that run together share less of dY in L2, which a
// list of many rounds does not win back.  Single calls on a cool chip, us, two launches and one: 8192 x 1024 x 50257 (a head) 1221, 1315;
// 4096 x 1024 x 50257 598, 604; 8192 x 2048 x 3072 187, 172; 8192 x 1024 x 4096 140, 121; 2048 x 1024 x 3072 79, 73.
static Plan choose(int rows, int in, int out, int want, int clusters) {
  struct Kept { int key[5]; Plan plan; };
  // sixteen sets of four, so that the layers of a model stay (with sizes that are multiples of a large power of two a sum of
  // multiples of them put all into one place, and each call of a block's four layers made its plan anew: 1.5 - 3 us of the host)
  static thread_local Kept kept[16][4];
  static thread_local unsigned char oldest[16];
  const int key[5] = {rows, in, out, want, clusters};
  uint32_t h = 0;
  for (int k : key) h = (h ^ (uint32_t)k) * 0x9e3779b1u, h ^= h >> 15;
  Kept* set = kept[h >> 28];
  for (int i = 0; i < 4; ++i)
    if (std::equal(key, key + 5, set[i].key)) return set[i].plan;
  Plan together{{{BN, 1}, {BN, 1}, {BN, 1}}, false}, apart{{{BN, 1}, {BN, 1}, {BN, 1}}, true};
  const long long one = best_list(rows, in, out, want, clusters, together.c);
  Kept& k = set[oldest[h >> 28]++ & 3];
  k.plan = together;
  if ((want & 3) == 3) {
    const long long two = best_list(rows, in, out, 1 << DX, clusters, apart.c) + best_list(rows, in, out, want & ~(1 << DX), clusters, apart.c);
    if (20 * one > 19 * (two + LAUNCH_CYCLES)) k.plan = apart;
  }
  std::copy(key, key + 5, k.key);
  return k.plan;
}

static int make_problem(int rows, int in, int out, int want, const Choice* c, Problem* p, size_t* ws_floats, int* counters) {
  p->parts = 0;
  for (int what = DX; what <= DW; ++what)
    if (want >> what & 1) set_part(&p->part[p->parts++], what, rows, in, out, c[what]);
  std::sort(p->part, p->part + p->parts, [](const Part& a, const Part& b) { return unit_cycles(a) > unit_cycles(b); });
  long long first = 0, ws = 0;
  int arrivals = 0;
  auto place = [&](Part& q) {
    const int tiles = q.tiles_m * q.tiles_n;
    q.first = (int)first;
    q.ws = ws;
    q.arrivals = arrivals;
    if (q.slices > 1) {
      ws += 2LL * tiles * q.slices * BM * (q.what == DB ? 1 : q.bn);
      arrivals += 2 * tiles;
    }
  };
  for (int i = 0; i < p->parts; ++i) {
    place(p->part[i]);
    first += (long long)p->part[i].tiles_m * p->part[i].tiles_n * p->part[i].slices;
  }
  if (want >> DB & 1) {
    set_part(&p->sums, DB, rows, in, out, c[DB]);
    place(p->sums);
  }
  p->total = (int)first;
  *ws_floats = std::max(*ws_floats, (size_t)ws);       // launches that follow each other share it
  *counters = std::max(*counters, arrivals);
  return TMPI_OK;
}

// The launches of a call: one or two.  form (0: chosen): columns / 64 and slices of dX, of dW, slices of db, four bits each from the
// lowest, then one bit for dX apart and two more for slices of db from 16.
static int plan(int rows, int in, int out, int want, int form, int clusters, Problem* p, int* launches, size_t* ws_floats, int* counters) {
  Plan c;
  if (form) {
    for (int what = DX; what <= DW; ++what) {
      c.c[what] = {64 * (form >> (8 * what) & 15), form >> (8 * what + 4) & 15};
      if (c.c[what].bn < 128 || c.c[what].bn > 256) return fail(TMPI_ERR_INVALID, "linear_bwd: form %#x", form);
    }
    c.c[DB] = {BN, (form >> 16 & 15) | (form >> 21 & 3) << 4};
    for (const Choice& x : c.c) if (x.slices < 1) return fail(TMPI_ERR_INVALID, "linear_bwd: form %#x", form);
    c.apart = (form >> 20 & 1) && (want & 3) == 3;
  } else {
    c = choose(rows, in, out, want, clusters);
  }
  *ws_floats = 0;
  *counters = 0;
  *launches = 0;
  if (c.apart) make_problem(rows, in, out, 1 << DX, c.c, &p[(*launches)++], ws_floats, counters);
  return make_problem(rows, in, out, c.apart ? want & ~(1 << DX) : want, c.c, &p[(*launches)++], ws_floats, counters);
}

}  // namespace lbwd
}  // namespace tmpi

using namespace tmpi;

extern "C" {

// What a call needs: bytes of workspace and arrival counters (unsigned, zero before the first call that uses them; every call leaves
// them zero).  want: 1 dX, 2 dW, 4 db, of which at least one of the first two.  Up to eight tiles of 256 KB for each cluster and product:
// none to 20 MB for most layers, 157 MB for 65536 x 256 x 50257.
int tmpi_linear_bwd_plan(int rows, int in, int out, int want, int form, size_t* workspace_bytes, int* counters) {
  if (rows < 1 || in < 1 || out < 1 || in % 8) return fail(TMPI_ERR_INVALID, "linear_bwd: stored rows must be multiples of 16 bytes (TMA)");
  if (!(want & 3) || want & ~7) return fail(TMPI_ERR_INVALID, "linear_bwd: nothing to compute");
  lbwd::Problem p[2] = {};
  size_t ws = 0;
  int launches;
  const int st = lbwd::plan(rows, in, out, want, form, lbwd::max_clusters(), p, &launches, &ws, counters);
  *workspace_bytes = ws * sizeof(float);
  return st;
}

// dx [rows, in] = dy w, dw [out, in] = dy^T x, db [out] = column sums of dy, for dy [rows, out] with rows ld_dy elements apart (0: dense;
// a multiple of 8, which out need not be), x [rows, in], w [out, in], all bf16 with fp32 accumulation; dx, dw, db may be null.
// Calls that share workspace or counters must not overlap.
int tmpi_linear_bwd(const void* dy, int64_t ld_dy, const void* x, const void* w, void* dx, void* dw, void* db, int rows, int in, int out, int form,
                    void* workspace, size_t workspace_bytes, void* counters, int ncounters, void* stream) {
  const int want = (dx ? 1 : 0) | (dw ? 2 : 0) | (db ? 4 : 0);
  if (!ld_dy) ld_dy = out;
  if (rows < 1 || in < 1 || out < 1 || in % 8 || ld_dy % 8 || ld_dy < out) return fail(TMPI_ERR_INVALID, "linear_bwd: stored rows must be multiples of 16 bytes (TMA)");
  if (!(want & 3)) return fail(TMPI_ERR_INVALID, "linear_bwd: nothing to compute");
  const int clusters = lbwd::max_clusters();
  lbwd::Problem p[2] = {};
  size_t ws = 0;
  int launches, need, st;
  if ((st = lbwd::plan(rows, in, out, want, form, clusters, p, &launches, &ws, &need))) return st;
  if ((ws && (!workspace || ((uintptr_t)workspace & 15))) || workspace_bytes < ws * sizeof(float) || ncounters < need || (need && !counters))
    return fail(TMPI_ERR_INVALID, "linear_bwd: workspace of %zu bytes (16-byte aligned) and %d counters needed", ws * sizeof(float), need);
  CUtensorMap mdy, mx, mw, mdx, mdw;
  if ((st = make_tmap_bf16(&mdy, dy, (uint64_t)rows, (uint64_t)out, (uint64_t)ld_dy, 64))) return st;
  mx = mw = mdx = mdw = mdy;
  if (dw && (st = make_tmap_bf16(&mx, x, (uint64_t)rows, (uint64_t)in, (uint64_t)in, 64))) return st;
  if (dx && (st = make_tmap_bf16(&mw, w, (uint64_t)out, (uint64_t)in, (uint64_t)in, 64))) return st;
  if (dx && (st = make_tmap_bf16(&mdx, dx, (uint64_t)rows, (uint64_t)in, (uint64_t)in, 64))) return st;
  if (dw && (st = make_tmap_bf16(&mdw, dw, (uint64_t)out, (uint64_t)in, (uint64_t)in, 64))) return st;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see pdl.cuh
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.blockDim = dim3(gemm2::GROUP_THREADS);
  cfg.dynamicSmemBytes = gemm2::SMEM_BYTES; cfg.stream = (cudaStream_t)stream; cfg.attrs = at; cfg.numAttrs = 2;
  for (int i = 0; i < launches; ++i) {
    p[i].ws = (float*)workspace;
    p[i].arrivals = (unsigned*)counters;
    p[i].dy = (const __nv_bfloat16*)dy;
    p[i].ld_dy = ld_dy;
    p[i].rows = rows;
    p[i].out = out;
    p[i].db = (__nv_bfloat16*)db;
    p[i].status = gemm_status_word();
    cfg.gridDim = dim3(2 * std::min(p[i].total + p[i].sums.tiles_m * p[i].sums.slices, clusters));
    const cudaError_t e = cudaLaunchKernelEx(&cfg, lbwd::linear_bwd_kernel, mdy, mx, mw, mdx, mdw, p[i]);
    if (e != cudaSuccess) return fail(TMPI_ERR_CUDA, "linear_bwd launch: %s", cudaGetErrorString(e));
  }
  return TMPI_OK;
}

}  // extern "C"
