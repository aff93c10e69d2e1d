// Causal self-attention backward (head size 64) as one tcgen05 kernel: dQ, dK, dV from Q, K, V, dO, the forward's
// log-sum-exp and delta = rowsum(dO * O).
//
// A work item is one block of 128 keys of one (batch, head); a persistent CTA per SM walks the query blocks of an item
// from its diagonal to the end of the sequence.  Scores are computed transposed, [key][query], so that P is born in
// the layout in which the tensor core takes its first operand out of tensor memory.  Per pair (query block i, key
// block j), five MMAs with fp32 accumulators in tensor memory:
//
//   S^T  = K_j Q_i^T          dP^T = V_j dO_i^T                     (128 keys x 128 queries each)
//   dV  += P^T dO_i                                                 (P^T read from tensor memory; 128 x 64)
//   dK  += dS^T Q_i           dQ_ij = dS K_j                        (dS^T read out of shared memory, K-major and MN-major; 128 x 64)
//
// with P = exp(scale S - lse) and dS = P (dP - delta); the softmax scale is applied to dK and dQ at the end.
//
//   warp 0      TMA producer: K_j and V_j through two buffers (the next item's arrive under the current one), Q_i, dO_i
//               and the block's 128 lse / delta values through a three-stage ring
//   warp 1      MMA issuer; order per pair n: S(n+1), dV(n), dP(n+1), dK(n), dQ(n), so that the exponentials of pair
//               n + 1 run under the products of pair n
//   warps 4-7   drain dQ_ij (every pair) and dK, dV (every item): one thread per row; dQ goes through a swizzled staging
//               tile and is added to the fp32 buffer by the TMA unit (cp.reduce, whole 128-byte rows), dK and dV are stored
//               through the same tiles (as 16-byte stores of 32 different rows they held up the next item for 2.5 us)
//   warps 8-23  four threads per key row: P^T as bf16 into its own tensor-memory columns, dS^T into shared memory, where both
//               dK and dQ read it: dP of the next pair need not wait until dK has read dS out of dP's columns
//
// What bounds it: neither the MMAs (about 1500 cycles per pair with their shared-memory operands) nor the 16384
// exponentials (1024 cycles), but the softmax warps' instructions and latencies, which fill the pair's 3500 cycles without a wait for
// the MMAs.  So nothing but two packed operations per pair of scores, the rounding and the stores lies there; masks are
// applied in the diagonal pair's own branch; a wait that succeeds does not look at the error word; waiting warps sleep.  Sixteen softmax
// warps share the work (eight: 105 us in place of 97).  Tried and taken back: half of the softmax warps offset by half a pair, so
// that the exponentials of some run beside the stores of the others (116 in place of 109); the statistics scaled by a warp of their
// own (100 in place of 96).  Measured on a B200, 8 x 16 heads x 1024 x 64, the three launches of a backward in a row: 113.5
// -> 90.5 us, of which this kernel 70; 1 x 16 x 2048 46.8 -> 39.5.
//
// The order in which CTAs add to dQ is not fixed, so its low bits vary; dK and dV are bit-reproducible.  Every wait is
// bounded; a CTA that gives up records where and frees its tensor memory.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <algorithm>
#include <mutex>
#include "sm100_ptx.cuh"
#include "attn_util.cuh"
#include "pdl.cuh"
#include "../include/tmpi_c_api.h"
#include "../runtime/common.h"

using namespace tmpi;

namespace tmpi {
int make_tmap_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
int make_tmap_f32(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
int gemm_sm_count();
}

namespace attnb {
using namespace attn_util;

constexpr int BLK = 128, D = 64, UMMA_K = 16, DRAIN_WARPS = 4, SOFTMAX_WARPS = 16;
constexpr int THREADS = 32 * (4 + DRAIN_WARPS + SOFTMAX_WARPS);
constexpr int QD_STAGES = 3;
constexpr int TILE = BLK * D * 2;                             // a 128 x 64 bf16 tile: 16 KB
constexpr int K_OFF = 0, V_OFF = 2 * TILE, Q_OFF = 4 * TILE, DO_OFF = Q_OFF + QD_STAGES * TILE,
              DS_OFF = DO_OFF + QD_STAGES * TILE, DQ_OFF = DS_OFF + 2 * TILE;
constexpr int SMEM_TILES = DQ_OFF + TILE;                     // 208 KB; the dQ staging is 4 KB (32 rows x 32 columns) per warp
constexpr int STAT_BYTES = BLK * 4;                           // lse or delta of a query block
constexpr int STAT_OFF = SMEM_TILES, SHARED_OFF = STAT_OFF + QD_STAGES * 2 * STAT_BYTES;
constexpr int SMEM_SHARED = 512, SMEM_BYTES = SHARED_OFF + SMEM_SHARED;
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
constexpr int TMEM_COLS = 512, T_S = 0, T_DP = 128, T_DV = 256, T_DK = 320, T_DQ = 384, T_P = 448;
constexpr unsigned long long kWaitBudgetNs = 2000000000ull;

struct alignas(128) Shared {
  uint64_t kv_full[2], kv_empty[2], qd_full[QD_STAGES], qd_empty[QD_STAGES], s_full, s_empty, p_full, dv_done, dp_full, ds_full,
      dq_full, dq_empty, acc_full, acc_empty;
  uint32_t tmem_base;
  int error;
};
static_assert(sizeof(Shared) <= SMEM_SHARED, "barrier block");

struct Params {
  int B, T, H, blocks, items;
  float scale, scale_log2;
  const float* lse;            // [B, H, T], natural log
  const float* delta;          // [B, H, T]
  int* status;
  unsigned long long* trace;   // optional: time stamps of the phases of CTA 0 (see tmpi_attention_bwd_set_trace)
};

__device__ __forceinline__ void fail(Shared* sh, const Params& p, int where) {
  atomicExch(&sh->error, where);
  if (p.status) atomicCAS(p.status, 0, 3100 + where);
}

// Phase time stamps of one CTA's first item for tuning: slot = (pair * 16 + event), written by one thread per role.
__device__ __forceinline__ void stamp(const Params& p, int round, int n, int ev) {
  if (p.trace && blockIdx.x == 0 && round == 0) p.trace[n * 16 + ev] = sm100::now_ns();
}

// The item of this CTA in a round: key blocks near the start of the sequence meet the most query blocks and come first,
// every other round in reverse, so that a CTA that got a long item gets a short one next.
__device__ __forceinline__ bool item(const Params& p, int round, int* bh, int* jblk) {
  const int g = (int)gridDim.x, i = (int)blockIdx.x;
  const long long t = (long long)round * g + ((round & 1) ? g - 1 - i : i);
  if (t >= p.items) return false;
  const int n = p.B * p.H;
  *jblk = (int)(t / n);
  *bh = (int)(t % n);
  return true;
}

// Position in a ring of N stages after every step over all items: stage index and the parity of its current use.
template <int N>
struct Ring {
  int stage = 0, use = 0;
  __device__ __forceinline__ void next() { if (++stage == N) { stage = 0; ++use; } }
};

#define ATTNB_WAIT(bar, parity, where) \
  do { if (!sm100::mbar_wait((bar), (parity), kWaitBudgetNs, &sh->error)) { fail(sh, p, (where)); return; } } while (0)
// In a whole warp the lanes go on, or leave, together: a wait may succeed for some of them and have run out for others, who would then be missing
// at the warp's next barrier.  A wait that has run out is noted, the lane goes on, with values that no longer matter, and the warp
// votes where its lanes meet anyway.
#define ATTNB_WARP_WAIT(bar, parity, where) \
  do { if (!sm100::mbar_wait((bar), (parity), kWaitBudgetNs, &sh->error)) { fail(sh, p, (where)); ok = false; } } while (0)

__device__ void producer(Shared* sh, unsigned char* smem, const Params& p, const CUtensorMap* mq, const CUtensorMap* mk,
                         const CUtensorMap* mv, const CUtensorMap* mdo) {
  Ring<QD_STAGES> q;
  int bh, jblk;
  for (int r = 0; item(p, r, &bh, &jblk); ++r) {
    const int b = bh / p.H, h = bh - b * p.H, row0 = b * p.T, kv = r & 1;
    if (r >= 2) ATTNB_WAIT(&sh->kv_empty[kv], ((r >> 1) - 1) & 1, 1);
    sm100::mbar_expect_tx(&sh->kv_full[kv], 2 * TILE);
    sm100::tma_load_2d(smem + K_OFF + kv * TILE, mk, h * D, row0 + jblk * BLK, &sh->kv_full[kv]);
    sm100::tma_load_2d(smem + V_OFF + kv * TILE, mv, h * D, row0 + jblk * BLK, &sh->kv_full[kv]);
    for (int i = jblk; i < p.blocks; ++i, q.next()) {
      const int st = q.stage;
      if (q.use >= 1) ATTNB_WAIT(&sh->qd_empty[st], (q.use - 1) & 1, 2);
      unsigned char* stat = smem + STAT_OFF + st * 2 * STAT_BYTES;
      const size_t at = (size_t)bh * p.T + (size_t)i * BLK;
      sm100::mbar_expect_tx(&sh->qd_full[st], 2 * TILE + 2 * STAT_BYTES);
      sm100::tma_load_2d(smem + Q_OFF + st * TILE, mq, h * D, row0 + i * BLK, &sh->qd_full[st]);
      sm100::bulk_load(stat, p.lse + at, STAT_BYTES, &sh->qd_full[st]);
      sm100::tma_load_2d(smem + DO_OFF + st * TILE, mdo, h * D, row0 + i * BLK, &sh->qd_full[st]);
      sm100::bulk_load(stat + STAT_BYTES, p.delta + at, STAT_BYTES, &sh->qd_full[st]);
    }
  }
}

__device__ void mma_issuer(Shared* sh, unsigned char* smem, const Params& p) {
  const uint32_t tm = sh->tmem_base;
  constexpr uint32_t idesc_s = sm100::make_idesc_f16(BLK, BLK, true);                 // both operands K-major
  constexpr uint32_t idesc_a = sm100::make_idesc_f16(BLK, D, true, true, false);      // A in tensor memory, B MN-major
  constexpr uint32_t idesc_q = sm100::make_idesc_f16(BLK, D, true, true, true);       // A and B MN-major
  // Descriptors: one per operand, built once; a slice or a stage further on only adds to the address field (bytes / 16 in
  // the low 14 bits; shared memory is far smaller than the field, so nothing carries out of it).
  auto at = [](uint64_t desc, uint32_t bytes) { return desc + (uint64_t)(bytes >> 4); };
  const uint64_t k_k = sm100::make_desc_sw128(sm100::smem_u32(smem + K_OFF)), v_k = sm100::make_desc_sw128(sm100::smem_u32(smem + V_OFF));
  const uint64_t q_k = sm100::make_desc_sw128(sm100::smem_u32(smem + Q_OFF)), do_k = sm100::make_desc_sw128(sm100::smem_u32(smem + DO_OFF));
  const uint64_t k_mn = sm100::make_desc_sw128_mn(sm100::smem_u32(smem + K_OFF), TILE, 1024);
  const uint64_t q_mn = sm100::make_desc_sw128_mn(sm100::smem_u32(smem + Q_OFF), TILE, 1024);
  const uint64_t do_mn = sm100::make_desc_sw128_mn(sm100::smem_u32(smem + DO_OFF), TILE, 1024);
  const uint64_t ds_mn = sm100::make_desc_sw128_mn(sm100::smem_u32(smem + DS_OFF), TILE, 1024);
  const uint64_t ds_k = sm100::make_desc_sw128(sm100::smem_u32(smem + DS_OFF));
  auto ready = [&](uint64_t* bar, int parity, int where) -> bool {
    if (sm100::mbar_wait(bar, parity & 1, kWaitBudgetNs, &sh->error)) return true;
    fail(sh, p, where);
    return false;
  };
  auto product_128 = [&](uint32_t d, uint64_t a, uint64_t b) {            // 128 x 128 over the 64 head columns
#pragma unroll
    for (int k = 0; k < D / UMMA_K; ++k)
      sm100::umma_f16(tm + d, at(a, k * UMMA_K * 2), at(b, k * UMMA_K * 2), idesc_s, k > 0 ? 1u : 0u);
  };
  int bh, jblk;
  if (!item(p, 0, &bh, &jblk)) return;
  if (!ready(&sh->kv_full[0], 0, 3) || !ready(&sh->qd_full[0], 0, 3)) return;
  sm100::tc_fence_after();
  product_128(T_S, k_k, q_k);
  sm100::umma_commit(&sh->s_full);
  product_128(T_DP, v_k, do_k);
  sm100::umma_commit(&sh->dp_full);
  Ring<QD_STAGES> q;                                       // the stage of the pair in work
  int g = 0;                                               // pairs done, over all items
  bool more = true;
  for (int r = 0; more; ++r) {
    const int pairs = p.blocks - jblk, kv = r & 1;
    more = item(p, r + 1, &bh, &jblk);
    for (int n = 0; n < pairs; ++n, ++g) {
      const bool last = n + 1 == pairs, next = !last || more;
      Ring<QD_STAGES> qn = q;
      qn.next();
      const int kvn = last ? (kv ^ 1) : kv;                // buffer of the next pair's K and V
      if (next) {                                          // S of the next pair, once this pair's has been read
        if (last && !ready(&sh->kv_full[kvn], (r + 1) >> 1, 3)) return;
        if (!ready(&sh->qd_full[qn.stage], qn.use, 4) || !ready(&sh->s_empty, g, 5)) return;
        stamp(p, r, n, 8);
        sm100::tc_fence_after();
        product_128(T_S, at(k_k, kvn * TILE), at(q_k, qn.stage * TILE));
        sm100::umma_commit(&sh->s_full);
        stamp(p, r, n, 9);
      }
      if (n == 0 && r > 0 && !ready(&sh->acc_empty, r - 1, 6)) return;    // the previous item's dK and dV have been read
      if (!ready(&sh->p_full, g, 7)) return;
      sm100::tc_fence_after();
#pragma unroll
      for (int k = 0; k < BLK / UMMA_K; ++k)               // dV += P^T dO: 16 queries = eight columns of packed P, 16 rows of dO
        sm100::umma_f16_tmem_a(tm + T_DV, tm + T_P + k * 8, at(do_mn, q.stage * TILE + k * UMMA_K * 128), idesc_a, (n | k) ? 1u : 0u);
      sm100::umma_commit(&sh->dv_done);
      if (!ready(&sh->ds_full, g, 8)) return;
      stamp(p, r, n, 10);
      sm100::tc_fence_after();
      if (next) {                                          // dP of the next pair: this pair's has been read
        product_128(T_DP, at(v_k, kvn * TILE), at(do_k, qn.stage * TILE));
        sm100::umma_commit(&sh->dp_full);
      }
#pragma unroll
      for (int k = 0; k < BLK / UMMA_K; ++k)               // dK += dS^T Q: 16 queries = 32 bytes of the rows of dS^T, 16 rows of Q
        sm100::umma_f16(tm + T_DK, at(ds_k, (k >> 2) * TILE + (k & 3) * UMMA_K * 2), at(q_mn, q.stage * TILE + k * UMMA_K * 128), idesc_a,
                        (n | k) ? 1u : 0u);
      sm100::umma_commit(&sh->qd_empty[q.stage]);          // every product that reads this stage is done
      if (last) sm100::umma_commit(&sh->acc_full);
      if (g > 0 && !ready(&sh->dq_empty, g - 1, 9)) return;
      sm100::tc_fence_after();
#pragma unroll
      for (int k = 0; k < BLK / UMMA_K; ++k)               // dQ_ij = dS K_j: 16 keys = 16 rows of dS^T and of K
        sm100::umma_f16(tm + T_DQ, at(ds_mn, k * UMMA_K * 128), at(k_mn, kv * TILE + k * UMMA_K * 128), idesc_q, k > 0 ? 1u : 0u);
      sm100::umma_commit(&sh->dq_full);                    // also: dS in shared memory is free again
      if (last) sm100::umma_commit(&sh->kv_empty[kv]);
      stamp(p, r, n, 12);
      q = qn;
    }
  }
}

// Four threads per key row (`part` picks 32 of the 128 queries of a pair).
__device__ void softmax_rows(Shared* sh, unsigned char* smem, const Params& p, int quarter, int part, int lane) {
  const int row = quarter * 32 + lane;                     // key inside the block; tensor-memory lane
  const uint32_t tm = sh->tmem_base + ((uint32_t)(quarter * 32) << 16);
  const uint32_t t_s = tm + T_S + part * 32, t_dp = tm + T_DP + part * 32, t_p = tm + T_P + part * 16;
  // this thread's first 16-byte unit in the swizzled row of dS; the other three differ from it in two bits of the address
  const uint32_t ds_unit = sm100::smem_u32(smem + DS_OFF + (part >> 1) * TILE + row * 128) + ((((part & 1) * 4) ^ (row & 7)) << 4);
  const unsigned long long c2x2 = pack2(__float_as_uint(p.scale_log2), __float_as_uint(p.scale_log2));
  const unsigned long long nl2e = pack2(__float_as_uint(-1.4426950408889634f), __float_as_uint(-1.4426950408889634f));
  const bool tracer = row == 0 && part == 0;
  bool ok = true;
  Ring<QD_STAGES> q;
  int g = 0, bh, jblk;
  for (int r = 0; item(p, r, &bh, &jblk); ++r) {
    const int pairs = p.blocks - jblk;
    for (int n = 0; n < pairs; ++n, ++g, q.next()) {
      const float4* lse = reinterpret_cast<const float4*>(smem + STAT_OFF + q.stage * 2 * STAT_BYTES) + part * 8;
      const float4* delta = lse + STAT_BYTES / 16;
      const bool diag = n == 0, masked = diag && part < quarter;               // masked: every query of the thread is before its key
      if (tracer) stamp(p, r, n, 0);
      ATTNB_WARP_WAIT(&sh->qd_full[q.stage], q.use & 1, 11);
      ATTNB_WARP_WAIT(&sh->s_full, g & 1, 12);
      if (tracer) stamp(p, r, n, 1);
      sm100::tc_fence_after();
      uint32_t s[32], w[16];
      sm100::tmem_ld_32x32(t_s, s);
      sm100::tmem_ld_wait();
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&sh->s_empty);     // S is in registers: the next pair's may overwrite it
      if (!masked) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {                      // P = exp2(S * scale * log2(e) - lse * log2(e)) over S in place
          const float4 l = lse[u];                         // the same four values for all lanes
          const unsigned long long l01 = mul2(pack2(__float_as_uint(l.x), __float_as_uint(l.y)), nl2e);
          const unsigned long long l23 = mul2(pack2(__float_as_uint(l.z), __float_as_uint(l.w)), nl2e);
          float a[4];
          unpack2(fma2(pack2(s[4 * u], s[4 * u + 1]), c2x2, l01), a[0], a[1]);
          unpack2(fma2(pack2(s[4 * u + 2], s[4 * u + 3]), c2x2, l23), a[2], a[3]);
#pragma unroll
          for (int e = 0; e < 4; ++e) s[4 * u + e] = __float_as_uint(ex2(a[e]));
        }
      }
      if (diag) {                                          // the diagonal block: queries before the key
#pragma unroll
        for (int e = 0; e < 32; ++e)
          if (part * 32 + e < row) s[e] = 0u;
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) w[e] = pack_bf16(s[2 * e], s[2 * e + 1]);
      if (g > 0) {                                         // dV of the previous pair has read P
        ATTNB_WARP_WAIT(&sh->dv_done, (g - 1) & 1, 13);
        sm100::tc_fence_after();
      }
      sm100::tmem_st_32x16(t_p, w);
      sm100::tmem_st_wait();
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&sh->p_full);
      ATTNB_WARP_WAIT(&sh->dp_full, g & 1, 14);
      sm100::tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {                        // dS = P (dP - delta), 16 queries at a time
        uint32_t d[16], v[8];
        sm100::tmem_ld_32x16(t_dp + c * 16, d);
        sm100::tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 dl = delta[c * 4 + u];
          const uint32_t* pv = &s[c * 16 + 4 * u];
          float a[4];
          unpack2(mul2(pack2(pv[0], pv[1]), sub2(pack2(d[4 * u], d[4 * u + 1]), pack2(__float_as_uint(dl.x), __float_as_uint(dl.y)))),
                  a[0], a[1]);
          unpack2(mul2(pack2(pv[2], pv[3]), sub2(pack2(d[4 * u + 2], d[4 * u + 3]), pack2(__float_as_uint(dl.z), __float_as_uint(dl.w)))),
                  a[2], a[3]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(a[2 * e], a[2 * e + 1]);
            v[2 * u + e] = *reinterpret_cast<uint32_t*>(&hh);
          }
        }
        if (masked) {                                      // dP - delta may be no number there
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = 0u;
        }
        if (c == 0 && g > 0) ATTNB_WARP_WAIT(&sh->dq_full, (g - 1) & 1, 15);          // dK and dQ of the previous pair have read dS
#pragma unroll
        for (int u = 0; u < 2; ++u)                        // eight queries = one 16-byte unit of the swizzled row
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                       ::"r"(ds_unit ^ ((c * 2 + u) << 4)), "r"(v[4 * u]), "r"(v[4 * u + 1]), "r"(v[4 * u + 2]), "r"(v[4 * u + 3]) : "memory");
      }
      sm100::fence_proxy_async_smem();                     // the MMA reads dS through the async proxy
      sm100::tc_fence_before();
      if (!__all_sync(~0u, ok)) return;
      if (lane == 0) {
        sm100::mbar_arrive(&sh->ds_full);
        sm100::mbar_arrive(&sh->qd_empty[q.stage]);        // the statistics have been read
      }
      if (tracer) stamp(p, r, n, 2);
    }
  }
}

// Reads dQ of every pair and dK, dV of every item; one thread per row of the tile.
__device__ void drain(Shared* sh, unsigned char* smem, const Params& p, const CUtensorMap* mdq, const CUtensorMap* mdk, const CUtensorMap* mdv,
                      int quarter, int lane) {
  const uint32_t tm = sh->tmem_base + ((uint32_t)(quarter * 32) << 16);
  unsigned char* staging = smem + DQ_OFF + quarter * (TILE / DRAIN_WARPS);      // 32 rows of 128 bytes
  const unsigned long long scale2 = pack2(__float_as_uint(p.scale), __float_as_uint(p.scale));
  const bool tracer = quarter == 0 && lane == 0;
  bool ok = true;
  auto scaled = [&](uint32_t (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float a0, a1;
      unpack2(mul2(pack2(v[i], v[i + 1]), scale2), a0, a1);
      v[i] = __float_as_uint(a0); v[i + 1] = __float_as_uint(a1);
    }
  };
  int g = 0, bh, jblk;
  for (int r = 0; item(p, r, &bh, &jblk); ++r) {
    const int pairs = p.blocks - jblk, b = bh / p.H, h = bh - b * p.H;
    uint32_t v[2][32];
    for (int n = 0; n < pairs; ++n, ++g) {
      if (tracer) stamp(p, r, n, 3);
      ATTNB_WARP_WAIT(&sh->dq_full, g & 1, 16);
      if (tracer) stamp(p, r, n, 4);
      sm100::tc_fence_after();
      sm100::tmem_ld_32x32(tm + T_DQ, v[0]);
      sm100::tmem_ld_32x32(tm + T_DQ + 32, v[1]);
      sm100::tmem_ld_wait();
      sm100::tc_fence_before();
      if (!__all_sync(~0u, ok)) return;
      if (lane == 0) sm100::mbar_arrive(&sh->dq_empty);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        scaled(v[c]);
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the staging tile has been read
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 8; ++u)
          *reinterpret_cast<uint4*>(staging + lane * 128 + ((u ^ (lane & 7)) << 4)) =
              make_uint4(v[c][4 * u], v[c][4 * u + 1], v[c][4 * u + 2], v[c][4 * u + 3]);
        sm100::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          sm100::tma_reduce_add_2d(mdq, staging, h * D + c * 32, b * p.T + (jblk + n) * BLK + quarter * 32);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      if (tracer) stamp(p, r, n, 5);
    }
    ATTNB_WARP_WAIT(&sh->acc_full, r & 1, 17);
    if (!__all_sync(~0u, ok)) return;
    sm100::tc_fence_after();
    auto store = [&](const CUtensorMap* map) {             // 32 rows of 64 bf16 through the staging tile
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = pack_bf16(v[u >> 2][(u & 3) * 8 + 2 * e], v[u >> 2][(u & 3) * 8 + 2 * e + 1]);
        *reinterpret_cast<uint4*>(staging + lane * 128 + ((u ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      sm100::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        sm100::tma_store_2d(map, staging, h * D, b * p.T + jblk * BLK + quarter * 32);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    };
    sm100::tmem_ld_32x32(tm + T_DV, v[0]);
    sm100::tmem_ld_32x32(tm + T_DV + 32, v[1]);
    sm100::tmem_ld_wait();
    store(mdv);
    sm100::tmem_ld_32x32(tm + T_DK, v[0]);
    sm100::tmem_ld_32x32(tm + T_DK + 32, v[1]);
    sm100::tmem_ld_wait();
    sm100::tc_fence_before();
    __syncwarp();
    if (lane == 0) sm100::mbar_arrive(&sh->acc_empty);
    scaled(v[0]);
    scaled(v[1]);
    store(mdk);
  }
  if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");     // every addition is done before the kernel ends
}

__global__ void __launch_bounds__(THREADS, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                     const __grid_constant__ CUtensorMap map_dq, const __grid_constant__ CUtensorMap map_dk,
                     const __grid_constant__ CUtensorMap map_dv, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Shared* sh = (Shared*)(smem_raw + SHARED_OFF);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && sm100::elect_one()) {
    sm100::tma_prefetch_desc(&map_q);
    sm100::tma_prefetch_desc(&map_k);
    sm100::tma_prefetch_desc(&map_v);
    sm100::tma_prefetch_desc(&map_do);
    sm100::tma_prefetch_desc(&map_dq);
    for (int s = 0; s < 2; ++s) { sm100::mbar_init(&sh->kv_full[s], 1); sm100::mbar_init(&sh->kv_empty[s], 1); }
    for (int s = 0; s < QD_STAGES; ++s) { sm100::mbar_init(&sh->qd_full[s], 1); sm100::mbar_init(&sh->qd_empty[s], 1 + SOFTMAX_WARPS); }
    sm100::mbar_init(&sh->s_full, 1);
    sm100::mbar_init(&sh->s_empty, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->p_full, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->dv_done, 1);
    sm100::mbar_init(&sh->dp_full, 1);
    sm100::mbar_init(&sh->ds_full, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->dq_full, 1);
    sm100::mbar_init(&sh->dq_empty, DRAIN_WARPS);
    sm100::mbar_init(&sh->acc_full, 1);
    sm100::mbar_init(&sh->acc_empty, DRAIN_WARPS);
    sh->error = 0;
    sm100::fence_barrier_init();
  }
  if (warp == 1) {
    sm100::tmem_alloc(&sh->tmem_base, TMEM_COLS);
    sm100::tmem_relinquish();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();

  wait_previous();
  const bool aligned = (sm100::smem_u32(smem_raw) & 1023u) == 0;     // the swizzled tiles need a 1024-byte aligned base
  if (!aligned) {
    if (threadIdx.x == 0) fail(sh, p, 18);
  } else if (warp < 4) {                                   // registers per four warps: 56 + 72 + 4 * 88 = the launch's 6 * 80
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      if (sm100::elect_one()) producer(sh, smem_raw, p, &map_q, &map_k, &map_v, &map_do);
    } else if (warp == 1) {
      if (sm100::elect_one()) mma_issuer(sh, smem_raw, p);
    }
  } else if (warp < 4 + DRAIN_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    drain(sh, smem_raw, p, &map_dq, &map_dk, &map_dv, warp & 3, lane);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
    softmax_rows(sh, smem_raw, p, warp & 3, (warp - 4 - DRAIN_WARPS) >> 2, lane);
  }
  __syncwarp();
  sm100::tc_fence_before();
  __syncthreads();
  if (sh->error && warp == 0 && sm100::elect_one()) {
    const unsigned long long t0 = sm100::now_ns();
    while (sm100::now_ns() - t0 < 200000000ull) { __nanosleep(1000); }   // copies in flight land within microseconds
  }
  __syncthreads();
  if (warp == 1) {
    sm100::tc_fence_after();
    sm100::tmem_dealloc(sh->tmem_base, TMEM_COLS);
  }
}

// The two passes around the main kernel are bound by the latency of their few dependent loads per thread.  Their indices are divided
// in 32 bits (there are below 2^32 of them: the fp32 dQ buffer alone would have 137 GB), which is a fraction of the
// instructions of a 64-bit division, and there are two rounds of blocks.  8 x 16 heads x 1024 x 64, the whole backward: 93.5 us with
// 64-bit divisions and half the blocks, 92.0 and 90.2 without.
constexpr int kPassBlocks = 148 * 16;

// delta[b, h, t] = sum_d dO[b, t, h, d] * O[b, t, h, d]: eight threads per (row, head), one 16-byte load of O and of
// dO each (a warp reads four whole 128-byte lines of each tensor per instruction), three shuffles; the same threads
// clear their 64 entries of the fp32 dQ buffer, so the caller need not.
__global__ void __launch_bounds__(256)
attention_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, int64_t ld_o, int64_t ld_do,
                       float* __restrict__ delta, float* __restrict__ dq_acc, int B, int T, int H) {
  wait_previous(o, dout);
  const long long total = (long long)B * T * H;                  // (row, head) pairs; blockDim.x / 8 of them per block and step
  const int sub = threadIdx.x & 7;
  for (long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3; idx < total;
       idx += ((long long)gridDim.x * blockDim.x) >> 3) {
    const unsigned r = (unsigned)idx / (unsigned)H;              // b * T + t
    const int h = (int)((unsigned)idx - r * (unsigned)H);
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(o + (size_t)r * ld_o + h * D) + sub);
    const uint4 g = __ldg(reinterpret_cast<const uint4*>(dout + (size_t)r * ld_do + h * D) + sub);
    const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wg[4] = {g.x, g.y, g.z, g.w};
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc = fmaf(__uint_as_float(wa[e] << 16), __uint_as_float(wg[e] << 16), acc);
      acc = fmaf(__uint_as_float(wa[e] & 0xffff0000u), __uint_as_float(wg[e] & 0xffff0000u), acc);
    }
    const unsigned group = 0xffu << (threadIdx.x & 24);          // the eight lanes of this (row, head)
    acc += __shfl_xor_sync(group, acc, 1);
    acc += __shfl_xor_sync(group, acc, 2);
    acc += __shfl_xor_sync(group, acc, 4);
    if (sub == 0) {
      const int b = (int)(r / (unsigned)T), t = (int)(r - (unsigned)b * (unsigned)T);
      delta[((size_t)b * H + h) * T + t] = acc;
    }
    float4* z = reinterpret_cast<float4*>(dq_acc + (size_t)r * (H * D) + h * D) + sub * 2;
    z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// dq[r, c] = bf16(dq_acc[r, c]): the fp32 sums of the reductions rounded into the Q block of the packed gradient.
__global__ void __launch_bounds__(256)
attention_dq_round_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, int64_t ld_dq, long long rows, int cols) {
  wait_previous(acc);
  const int groups = cols / 8;
  const long long total = rows * groups;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
    const long long r = (unsigned)idx / (unsigned)groups;
    const int c = (int)((unsigned)idx - (unsigned)r * (unsigned)groups) * 8;
    const float4 a = *reinterpret_cast<const float4*>(acc + r * cols + c), b = *reinterpret_cast<const float4*>(acc + r * cols + c + 4);
    __nv_bfloat162 h0 = __floats2bfloat162_rn(a.x, a.y), h1 = __floats2bfloat162_rn(a.z, a.w);
    __nv_bfloat162 h2 = __floats2bfloat162_rn(b.x, b.y), h3 = __floats2bfloat162_rn(b.z, b.w);
    uint4 u;
    u.x = *reinterpret_cast<uint32_t*>(&h0); u.y = *reinterpret_cast<uint32_t*>(&h1);
    u.z = *reinterpret_cast<uint32_t*>(&h2); u.w = *reinterpret_cast<uint32_t*>(&h3);
    *reinterpret_cast<uint4*>(dq + r * ld_dq + c) = u;
  }
}

}  // namespace attnb

static unsigned long long* g_attnb_trace = nullptr;

static int* attnb_status_word(int** host_out = nullptr) {
  static int* dev_ptr = nullptr;
  static int* host_ptr = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    if (cudaHostAlloc((void**)&host_ptr, sizeof(int), cudaHostAllocMapped) == cudaSuccess) {
      *host_ptr = 0;
      cudaHostGetDevicePointer((void**)&dev_ptr, host_ptr, 0);
    }
  });
  if (host_out) *host_out = host_ptr;
  return dev_ptr;
}

extern "C" {

// Gradients of tmpi_attention_fwd.  q, k, v as there (common row pitch ld_qkv); o and dout are [B * T, H * 64] with
// their own pitches; lse [B, H, T] from the forward; delta [B, H, T] is scratch (written here); dq_acc is a fp32
// [B * T, H * 64] buffer (cleared here) that receives dQ; dq (optional), dk and dv are bf16 [B * T, ld_dkv] (for instance
// the column blocks of the gradient of a packed QKV projection): dk and dv are written by the main kernel, dq by a last
// pass that rounds dq_acc.
int tmpi_attention_bwd(const void* q, const void* k, const void* v, int64_t ld_qkv, const void* o, int64_t ld_o,
                       const void* dout, int64_t ld_do, const float* lse, float* delta, float* dq_acc, void* dq, void* dk,
                       void* dv, int64_t ld_dkv, int B, int T, int H, float scale, void* stream) {
  if (B < 1 || H < 1 || T < 128 || T % 128) return fail(TMPI_ERR_UNSUPPORTED, "attention backward: T=%d must be a positive multiple of 128", T);
  if (ld_dkv % 8 || ((uintptr_t)dk & 15) || ((uintptr_t)dv & 15) || ((uintptr_t)dq_acc & 15) || ld_o % 8 || ld_do % 8 ||
      ((uintptr_t)o & 15) || ((uintptr_t)dout & 15) || ((uintptr_t)lse & 15) || ((uintptr_t)delta & 15))
    return fail(TMPI_ERR_INVALID, "attention backward: operands must be 16-byte aligned with pitches that are multiples of 8");
  if ((int64_t)B * H * (T / 128) > 0x7fffffffLL) return fail(TMPI_ERR_INVALID, "attention backward: too many blocks");
  cudaStream_t s = (cudaStream_t)stream;
  const long long rows_heads = (long long)B * T * H;
  const int dgrid = (int)std::min<long long>((rows_heads * 8 + 255) / 256, attnb::kPassBlocks);
  cudaError_t e = launch_overlapped(attnb::attention_delta_kernel, dgrid, 256, 0, s, (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout,
                                    ld_o, ld_do, delta, dq_acc, B, T, H);
  if (e != cudaSuccess) return fail(TMPI_ERR_CUDA, "attention backward launch: %s", cudaGetErrorString(e));
  CUtensorMap mq, mk, mv, mdo, mdq, mdk, mdv;
  int st;
  const uint64_t rows = (uint64_t)B * T, cols = (uint64_t)H * attnb::D;
  if ((st = make_tmap_bf16(&mq, q, rows, cols, (uint64_t)ld_qkv, 128))) return st;
  if ((st = make_tmap_bf16(&mk, k, rows, cols, (uint64_t)ld_qkv, 128))) return st;
  if ((st = make_tmap_bf16(&mv, v, rows, cols, (uint64_t)ld_qkv, 128))) return st;
  if ((st = make_tmap_bf16(&mdo, dout, rows, cols, (uint64_t)ld_do, 128))) return st;
  if ((st = make_tmap_f32(&mdq, dq_acc, rows, cols, cols, 32))) return st;
  if ((st = make_tmap_bf16(&mdk, dk, rows, cols, (uint64_t)ld_dkv, 32))) return st;
  if ((st = make_tmap_bf16(&mdv, dv, rows, cols, (uint64_t)ld_dkv, 32))) return st;
  const int smem = attnb::SMEM_BYTES;
  cudaError_t ae = cudaFuncSetAttribute(attnb::attention_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (ae != cudaSuccess) return fail(TMPI_ERR_CUDA, "attention backward: shared memory attribute: %s", cudaGetErrorString(ae));
  attnb::Params p;
  p.B = B; p.T = T; p.H = H; p.blocks = T / attnb::BLK;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = lse; p.delta = delta;
  p.status = attnb_status_word();
  p.trace = g_attnb_trace;
  p.items = B * H * p.blocks;
  e = launch_overlapped(attnb::attention_bwd_kernel, std::min(p.items, gemm_sm_count()), attnb::THREADS, smem, s, mq, mk, mv, mdo, mdq, mdk, mdv, p);
  if (dq && e == cudaSuccess) {
    if ((uintptr_t)dq & 15) return fail(TMPI_ERR_INVALID, "attention backward: dq must be 16-byte aligned");
    const long long groups = (long long)rows * (cols / 8);
    const int cgrid = (int)std::min<long long>((groups + 255) / 256, attnb::kPassBlocks);
    e = launch_overlapped(attnb::attention_dq_round_kernel, cgrid, 256, 0, s, dq_acc, (__nv_bfloat16*)dq, ld_dkv, (long long)rows, (int)cols);
  }
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "attention backward launch: %s", cudaGetErrorString(e));
}

// Tuning aid: with a device buffer of (T / 128) * 16 64-bit words, CTA 0 of every later launch (the first key block of
// the first batch and head, which meets every query block) records the time of each phase of each pair (ns):
// 0 waits for S, 1 has it, 2 dS announced, 3 waits for dQ, 4 has it, 5 additions issued; MMA thread: 8 S was read and the
// next tiles are there, 9 next S issued, 10 has dS, 12 three products issued.
void tmpi_attention_bwd_set_trace(void* device_buffer) { g_attnb_trace = (unsigned long long*)device_buffer; }

// Non-zero after a CTA of the attention backward gave up on a bounded wait (3100 + the point where); clears it.
int tmpi_attention_bwd_status(void) {
  int* host = nullptr;
  attnb_status_word(&host);
  if (!host) return 0;
  int v = *(volatile int*)host;
  if (v) *(volatile int*)host = 0;
  return v;
}

}  // extern "C"
