// Causal self-attention forward (softmax(Q K^T / sqrt(d)) V, head size 64) as one tcgen05 kernel.
//
// The reference has no attention (its models are MNIST networks, examples/mnist/*.lua); the GPT-2 configuration
// of this package needs one, and it is a contraction, so it belongs on the tensor cores.  Work items are blocks of
// 128 queries of one (batch, head); a CTA walks the key / value blocks of an item up to its diagonal:
//
//   one warp    TMA producer: Q tiles through two buffers (the next item's Q is fetched under the current one), K and V
//               tiles of 128 keys through two-stage rings
//   one warp    MMA issuer:   S = Q K^T (128 x 128, fp32, tensor memory), then O += P V (128 x 64) with P read from
//               tensor memory and O accumulated there over all key blocks
//   eight warps softmax:     two threads per query row, 64 scores each (tcgen05.ld 32x32b gives a thread its own row, so
//                            there are no shuffles; the halves exchange their maxima through shared memory): the scores
//                            go into registers at once, which frees S for the next block's MMA; maximum, P = exp2(scaled
//                            S - m) as bf16 into tensor memory
//
// What bounds it: neither the special-function unit (16 exp2 per cycle and SM, 1024 cycles per 128 x 128 block; a quarter of
// them run as a cubic on the FMA pipe) nor the MMAs (512 cycles per block), but the latency of a team's chain S -> maximum
// -> P -> P V, about 1.6 us per key block.  Everything that is not needed per score is therefore kept off the softmax
// warps: P goes to tensor memory (no shared-memory stores, swizzle arithmetic or proxy fence), and O stays in tensor
// memory: only where a row's maximum grew do its threads scale O there by exp2(old max - new max), instead of reading every
// O_j back.  Tried and taken back: moving the maximum only when it grows by more than 2^8 (the largest P of a row is then
// no longer exactly 1, and its bf16 rounding showed in the output); one thread per row (63 us in place of 56); all
// exponentials before the wait for the previous product (61); descriptors in uniform registers (no difference); an item's output
// written inside the next one's first block (no faster, 34 in place of 22 us where the teams share items: registers).
//
// A CTA (one per SM) runs two such teams, each with its own rings, barriers and 256 tensor-memory columns, so that
// one exponentiates while the other waits.  Each has items of its own, or, where there are few, both work on the same one, on half
// of its key blocks each (attention_shares).  Teams are persistent and take items longest-first in snake order (item
// r * G + i, then r * G + G - 1 - i), which leaves the key blocks per team within one of each other at 8 x 16 x 1024; the
// next item's loads and first S run under the end of the current one.
//
// Measured on a B200, launches in a row: 8 x 16 heads x 1024 x 64 39.6 us, 1 x 16 x 2048 20.8 (47.7 and 25.5 before waiting warps
// slept, waits looked at the error word only when they do not succeed, and the halves met at named barriers).
//
// Q, K and V are read where the fused QKV projection left them ([B * T, 3 C], one tensor map per operand) and the
// output is written as [B * T, C]: no transposes around the kernel.  Every wait is bounded; a CTA that gives up records
// where in the status word and frees its tensor memory.
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
int gemm_sm_count();
}

namespace attn {
using namespace attn_util;

constexpr int BQ = 128, BKV = 128, D = 64, TEAMS = 2, SOFTMAX_WARPS = 8, UMMA_K = 16;
constexpr int THREADS = 32 * TEAMS * (2 + SOFTMAX_WARPS);
constexpr int TILE_BYTES = 128 * D * 2;                       // a 128 x 64 bf16 tile: 16 KB
constexpr int Q_OFF = 0, K_OFF = 2 * TILE_BYTES, V_OFF = 4 * TILE_BYTES, SMEM_TILES = 6 * TILE_BYTES;
constexpr int SMEM_SHARED = 256;                              // the teams' barrier blocks follow their tiles
constexpr int XCH_BYTES = 2 * 2 * BQ * 4;                     // two phases x two halves of the rows: values the halves exchange
constexpr int MERGE_BYTES = 2 * BQ * 4;                       // team 1's row maxima and sums of an item that the teams share
constexpr int SMEM_BYTES = TEAMS * (SMEM_TILES + SMEM_SHARED + XCH_BYTES) + MERGE_BYTES;
constexpr int TMEM_COLS = 256, TMEM_P = 128, TMEM_O = 192;    // S: columns 0-127 of a team, P (bf16 pairs): 128-191, O: 192-255
constexpr float LOWEST = -3.402823466e38f;
constexpr unsigned long long kWaitBudgetNs = 2000000000ull;

struct alignas(128) Shared {
  uint64_t q_full[2], q_empty[2], k_full[2], k_empty[2], v_full[2], v_empty[2], s_full, s_empty, p_full, pv_done, o_empty;
  uint64_t merge_full, merge_empty;      // of team 1, where the teams share items: its row sums are there, have been read
  uint32_t tmem_base;
  int error;
};
static_assert(sizeof(Shared) <= SMEM_SHARED, "barrier block");

struct Params {
  int B, T, H, q_blocks, items;
  float scale_log2;            // softmax scale times log2(e)
  __nv_bfloat16* out;          // [B * T, ld_out], head h at columns h * 64
  int ld_out;
  float* lse;                  // [B, H, T]: natural-log sum of exponentials of the scaled scores
  int* status;
  unsigned long long* trace;   // optional: time stamps of the phases of CTA 0 (see tmpi_attention_set_trace)
};

__device__ __forceinline__ void fail(Shared* sh, const Params& p, int where) {
  atomicExch(&sh->error, where);
  if (p.status) atomicCAS(p.status, 0, 3000 + where);
}

// Warps 0-1 are the producers of the two teams, 2-3 the MMA issuers, 4-11 and 12-19 the softmax warps.
__device__ __forceinline__ int team() {
  const int warp = threadIdx.x >> 5;
  return warp < 4 ? warp & 1 : (warp - 4) / SOFTMAX_WARPS;
}

// Phase time stamps of one team's first item for tuning: slot = (block * 16 + event), written by one thread per role.
__device__ __forceinline__ void stamp(const Params& p, int round, int j, int ev) {
  if (p.trace && blockIdx.x == 0 && round == 0 && team() == 0) p.trace[j * 16 + ev] = sm100::now_ns();
}

// The items of a team one after the other: (batch, head), query block and the key blocks [first, end) of it that are the
// team's.  Long items (late query blocks) first, every other round in reverse so that a team that got a long item gets a short
// one next.  SHARED: the CTA is the unit; team 0 takes the first half of an item's key blocks, team 1 the rest up to the
// diagonal (nothing of an item of one block).
template <bool SHARED> struct Items {
  int round = -1, bh, qblk, first, end;
  __device__ __forceinline__ bool next(const Params& p) {
    const unsigned g = SHARED ? gridDim.x : TEAMS * gridDim.x, i = blockIdx.x + (SHARED ? 0u : team() * gridDim.x), n = p.B * p.H;
    do {
      ++round;
      const unsigned t = round * g + ((round & 1) ? g - 1 - i : i);        // below 2^31 and one round more
      if (t >= (unsigned)p.items) return false;
      qblk = p.q_blocks - 1 - (int)(t / n);
      bh = (int)(t % n);
      const int half = (qblk + 2) >> 1;
      first = SHARED && team() ? half : 0;
      end = SHARED && !team() ? half : qblk + 1;
    } while (SHARED && first == end);
    return true;
  }
};

#define ATTN_WAIT(bar, parity, where) \
  do { if (!sm100::mbar_wait((bar), (parity), kWaitBudgetNs, &sh->error)) { fail(sh, p, (where)); return; } } while (0)

template <bool SHARED>
__device__ void producer(Shared* sh, unsigned char* tiles, const Params& p, const CUtensorMap* mq, const CUtensorMap* mk,
                         const CUtensorMap* mv) {
  int kc = 0, vc = 0;                                      // K and V tiles loaded so far, over all items
  Items<SHARED> it;
  for (int r = 0; it.next(p); ++r) {
    const int b = it.bh / p.H, h = it.bh - b * p.H, row0 = b * p.T;
    auto load_k = [&](int j) -> bool {
      const int st = kc & 1;
      if (kc >= 2 && (!sm100::mbar_wait(&sh->k_empty[st], ((kc >> 1) - 1) & 1, kWaitBudgetNs, &sh->error))) return false;
      sm100::mbar_expect_tx(&sh->k_full[st], TILE_BYTES);
      sm100::tma_load_2d(tiles + K_OFF + st * TILE_BYTES, mk, h * D, row0 + j * BKV, &sh->k_full[st]);
      ++kc;
      return true;
    };
    if (r >= 2) ATTN_WAIT(&sh->q_empty[r & 1], ((r >> 1) - 1) & 1, 12);
    sm100::mbar_expect_tx(&sh->q_full[r & 1], TILE_BYTES);
    sm100::tma_load_2d(tiles + Q_OFF + (r & 1) * TILE_BYTES, mq, h * D, row0 + it.qblk * BQ, &sh->q_full[r & 1]);
    if (!load_k(it.first)) { fail(sh, p, 1); return; }
    for (int j = it.first; j < it.end; ++j) {
      if (j + 1 < it.end && !load_k(j + 1)) { fail(sh, p, 1); return; }          // K runs one block ahead of V
      const int st = vc & 1;
      if (vc >= 2) ATTN_WAIT(&sh->v_empty[st], ((vc >> 1) - 1) & 1, 13);
      sm100::mbar_expect_tx(&sh->v_full[st], TILE_BYTES);
      sm100::tma_load_2d(tiles + V_OFF + st * TILE_BYTES, mv, h * D, row0 + j * BKV, &sh->v_full[st]);
      ++vc;
    }
  }
}

template <bool SHARED>
__device__ void mma_issuer(Shared* sh, unsigned char* tiles, const Params& p) {
  const uint32_t tmem_s = sh->tmem_base, tmem_p = sh->tmem_base + TMEM_P, tmem_o = sh->tmem_base + TMEM_O;
  constexpr uint32_t idesc_s = sm100::make_idesc_f16(BQ, BKV, true);            // Q and K both K-major
  constexpr uint32_t idesc_o = sm100::make_idesc_f16(BQ, D, true, true);        // P in tensor memory, V MN-major (d contiguous)
  const uint64_t dq = sm100::make_desc_sw128(sm100::smem_u32(tiles + Q_OFF));
  const uint64_t dk = sm100::make_desc_sw128(sm100::smem_u32(tiles + K_OFF));
  const uint64_t dv = sm100::make_desc_sw128_mn(sm100::smem_u32(tiles + V_OFF), TILE_BYTES, 1024);
  // a slice further into shared memory only adds to the address field (bytes / 16 in the low 14 bits)
  auto at = [](uint64_t desc, uint32_t bytes) { return desc + (uint64_t)(bytes >> 4); };
  int g = 0;                                               // key blocks whose S has been issued, over all items
  // S of a key block of this team's r-th item (block number g): waits for the softmax warps to have read the previous S
  auto issue_s = [&](int r, bool first, bool last) -> bool {
    if (first && (!sm100::mbar_wait(&sh->q_full[r & 1], (r >> 1) & 1, kWaitBudgetNs, &sh->error))) return false;
    if (!sm100::mbar_wait(&sh->k_full[g & 1], (g >> 1) & 1, kWaitBudgetNs, &sh->error)) return false;
    if (g >= 1 && (!sm100::mbar_wait(&sh->s_empty, (g - 1) & 1, kWaitBudgetNs, &sh->error))) return false;
    sm100::tc_fence_after();
    const uint64_t a = at(dq, (r & 1) * TILE_BYTES), b = at(dk, (g & 1) * TILE_BYTES);
#pragma unroll
    for (int k = 0; k < D / UMMA_K; ++k)
      sm100::umma_f16(tmem_s, at(a, k * UMMA_K * 2), at(b, k * UMMA_K * 2), idesc_s, k > 0 ? 1u : 0u);
    sm100::umma_commit(&sh->s_full);
    sm100::umma_commit(&sh->k_empty[g & 1]);
    if (last) sm100::umma_commit(&sh->q_empty[r & 1]);
    ++g;
    return true;
  };
  Items<SHARED> it;
  bool more = it.next(p);
  if (more && !issue_s(0, true, it.end - it.first == 1)) { fail(sh, p, 3); return; }
  int v = 0;                                               // P V products issued so far
  for (int r = 0; more; ++r) {
    const int first = it.first, last = it.end - 1;
    more = it.next(p);                                     // the next item: its first S runs before this one's last P V
    for (int j = first; j <= last; ++j) {
      if (j < last) {
        stamp(p, r, j, 8);
        if (!issue_s(r, false, j + 1 == last)) { fail(sh, p, 4); return; }
        stamp(p, r, j, 9);
      } else if (more) {
        if (!issue_s(r + 1, true, it.end - it.first == 1)) { fail(sh, p, 5); return; }
      }
      if (j == first && r > 0) ATTN_WAIT(&sh->o_empty, (r - 1) & 1, 14);       // the previous item's output has been read
      ATTN_WAIT(&sh->p_full, v & 1, 6);
      stamp(p, r, j, 10);
      ATTN_WAIT(&sh->v_full[v & 1], (v >> 1) & 1, 15);
      stamp(p, r, j, 11);
      sm100::tc_fence_after();
      const uint64_t b = at(dv, (v & 1) * TILE_BYTES);
#pragma unroll
      for (int k = 0; k < BKV / UMMA_K; ++k)               // 16 keys: eight columns of packed P, 16 rows of V
        sm100::umma_f16_tmem_a(tmem_o, tmem_p + k * (UMMA_K / 2), at(b, k * UMMA_K * 128), idesc_o, (j > first || k) ? 1u : 0u);
      sm100::umma_commit(&sh->pv_done);
      sm100::umma_commit(&sh->v_empty[v & 1]);
      stamp(p, r, j, 12);
      ++v;
    }
  }
}

// Scores s[0, 32) of one row (a chunk of 32 keys) -> sixteen packed bf16 pairs of exp2(s * c2 + nmc), added to the row
// sums.  A quarter of the exponentials run on the FMA pipe, the rest on the special-function unit; a masked score (-inf)
// gives exactly 0 on both.
__device__ __forceinline__ void exp_chunk(const uint32_t (&s)[32], uint32_t (&w)[16], unsigned long long c2x2,
                                          unsigned long long nmc2, unsigned long long& sum2) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float a0, a1;
    unpack2(fma2(pack2(s[2 * i], s[2 * i + 1]), c2x2, nmc2), a0, a1);
    const unsigned long long e = (i & 3) == 3 ? ex2_fma2(a0, a1) : pack2(__float_as_uint(ex2(a0)), __float_as_uint(ex2(a1)));
    sum2 = add2(sum2, e);
    float e0, e1;
    unpack2(e, e0, e1);
    w[i] = pack_bf16(__float_as_uint(e0), __float_as_uint(e1));
  }
}

// The two warps that share 32 rows meet at a named barrier (an mbarrier between them: 42.3 us in place of 40.8 at 8 x 16 x 1024, 22.1 in
// place of 20.9 for 1 x 16 x 2048).  A warp that gives up sets the error word and arrives there once more, so that its partner is
// not left waiting.  The partner then ends at its next s_full or pv_done, which need all warps; only at the end of an item does it come
// here twice without such a wait, and looks at the word in between.
__device__ __forceinline__ void pair_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(1 + team() * 4 + quarter) : "memory"); }
__device__ __forceinline__ void pair_leave(int quarter) { asm volatile("bar.arrive %0, 64;" ::"r"(1 + team() * 4 + quarter) : "memory"); }
#define ROWS_WAIT(bar, parity, where) \
  do { if (!sm100::mbar_wait_warp((bar), (parity), kWaitBudgetNs, &sh->error)) { fail(sh, p, (where)); __syncwarp(); pair_leave(quarter); return; } } while (0)

// Two threads per query row: `half` picks 64 of the 128 scores of a block and 32 of the 64 output columns.  The halves
// exchange their maxima through shared memory, block by block, and their row sums at the end of an item.
template <bool SHARED>
__device__ void softmax_rows(Shared* sh, Shared* other_team, float* xch, float2* merge, const Params& p, int quarter, int half, int lane) {
  const int row = quarter * 32 + lane;                     // the row of the tile; its tensor-memory lane
  const uint32_t tmem = sh->tmem_base + ((uint32_t)(quarter * 32) << 16);
  const uint32_t tmem_s = tmem + half * 64, tmem_p = tmem + TMEM_P + half * 32, tmem_o = tmem + TMEM_O + half * 32;
  const float c2 = p.scale_log2;
  const unsigned long long c2x2 = pack2(__float_as_uint(c2), __float_as_uint(c2));
  const bool tracer = row == 0 && half == 0;
  int g = 0, met = 0, merged = 0;                          // key blocks done, exchanges made and items merged so far
  // this row's value of the other half
  auto exchange = [&](float v, float* other) {
    float* x = xch + (met & 1) * 2 * BQ;
    x[half * BQ + row] = v;
    pair_sync(quarter);
    *other = x[(half ^ 1) * BQ + row];
    ++met;
  };
  Items<SHARED> it;
  for (int r = 0; it.next(p); ++r) {
    float m = -INFINITY;                                   // the running maximum
    unsigned long long sum2[2] = {0ull, 0ull};
    for (int j = it.first; j < it.end; ++j, ++g) {
      const bool diag = j == it.qblk;
      uint32_t s[2][32];
      if (tracer) stamp(p, r, j, 0);
      ROWS_WAIT(&sh->s_full, g & 1, 7);
      if (tracer) stamp(p, r, j, 1);
      sm100::tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) sm100::tmem_ld_32x32(tmem_s + c * 32, s[c]);
      sm100::tmem_ld_wait();
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&sh->s_empty);     // S is in registers: the next S may overwrite it
      if (diag) {                                          // keys after the query
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int chunk = half * 2 + c;
          if (chunk >= quarter) {                          // warp-uniform
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (chunk > quarter || i > lane) s[c][i] = 0xff800000u;
          }
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;      // four chains
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        mx0 = max3_nan(mx0, __uint_as_float(s[0][i]), __uint_as_float(s[0][i + 1]));
        mx1 = max3_nan(mx1, __uint_as_float(s[0][i + 2]), __uint_as_float(s[0][i + 3]));
        mx2 = max3_nan(mx2, __uint_as_float(s[1][i]), __uint_as_float(s[1][i + 1]));
        mx3 = max3_nan(mx3, __uint_as_float(s[1][i + 2]), __uint_as_float(s[1][i + 3]));
      }
      float mx = max_nan(max3_nan(mx0, mx1, mx2), mx3), mx_other;
      exchange(mx, &mx_other);
      mx = max_nan(mx, mx_other);
      if (tracer) stamp(p, r, j, 2);
      // the running maximum; where it grew, O and l so far are scaled by alpha (1 for rows where it did not)
      const float next = max_nan(m, mx);
      const bool grew = j > it.first && __any_sync(~0u, next > m);
      // While every key has scored -inf, scores are taken relative to a finite value: those keys weigh 0, wherever they lie.  (One
      // instruction with an immediate: a comparison and a selection, or a bound from the parameters, cost 8 x 16 x 1024 a
      // microsecond of 49.4.  LOWEST * c2 is finite for scales up to ln 2; a steeper one is not given shared items, and keys that
      // score -inf throughout the first block still make a row NaN there.)
      const float base = max_nan(next, LOWEST);
      const float alpha = ex2((m - base) * c2);
      const unsigned long long al2 = pack2(__float_as_uint(alpha), __float_as_uint(alpha));
      m = next;
      if (grew) { sum2[0] = mul2(sum2[0], al2); sum2[1] = mul2(sum2[1], al2); }
      // NaN where the maximum is NaN or +inf, and with it every P of the row: the polynomial's clamp alone would drop a NaN
      const float nmc = fmaf(base, 0.f, -base * c2);
      const unsigned long long nmc2 = pack2(__float_as_uint(nmc), __float_as_uint(nmc));
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[16], o[2][16];
        if (diag && half * 2 + c > quarter) {              // every key of the chunk is after every query of the warp
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = 0u;
        } else {
          exp_chunk(s[c], w, c2x2, nmc2, sum2[c]);
        }
        if (c == 0 && g > 0) {     // the previous block's product has read its P and added to O
          ROWS_WAIT(&sh->pv_done, (g - 1) & 1, 8);
          if (tracer && j > it.first) { stamp(p, r, j - 1, 5); stamp(p, r, j - 1, 6); }
          sm100::tc_fence_after();
        }
        sm100::tmem_st_32x16(tmem_p + c * 16, w);
        if (c == 1 && grew) {                              // the scores are spent: their registers hold O
          sm100::tmem_ld_32x16(tmem_o, o[0]);
          sm100::tmem_ld_32x16(tmem_o + 16, o[1]);
          sm100::tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              float a0, a1;
              unpack2(mul2(pack2(o[q][i], o[q][i + 1]), al2), a0, a1);
              o[q][i] = __float_as_uint(a0); o[q][i + 1] = __float_as_uint(a1);
            }
            sm100::tmem_st_32x16(tmem_o + q * 16, o[q]);
          }
        }
      }
      sm100::tmem_st_wait();
      if (tracer) stamp(p, r, j, 3);
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&sh->p_full);
      if (tracer) stamp(p, r, j, 4);
    }
    // the item's output: O / l
    float l0, l1, l_other;
    unpack2(add2(sum2[0], sum2[1]), l0, l1);
    if (__any_sync(~0u, *(volatile int*)&sh->error)) { pair_leave(quarter); return; }     // the partner may have left at the last exchange
    exchange(l0 + l1, &l_other);
    float l = half ? l_other + (l0 + l1) : (l0 + l1) + l_other;
    const bool merges = SHARED && it.qblk > 0;
    if (merges && team()) {                                // hand over O (in tensor memory), maximum and sum; go on
      if (merged > 0) ROWS_WAIT(&sh->merge_empty, (merged - 1) & 1, 16);
      if (half == 0) merge[row] = make_float2(m, l);
      ROWS_WAIT(&sh->pv_done, (g - 1) & 1, 10);
      sm100::tc_fence_after();
      sm100::tc_fence_before();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&sh->merge_full);
      ++merged;
      continue;
    }
    float inv = 1.f / l;
    ROWS_WAIT(&sh->pv_done, (g - 1) & 1, 10);
    if (tracer) stamp(p, r, it.qblk, 5);
    sm100::tc_fence_after();
    uint32_t o[32];
    sm100::tmem_ld_32x32(tmem_o, o);
    sm100::tmem_ld_wait();
    if (merges) {
      ROWS_WAIT(&other_team->merge_full, merged & 1, 17);
      ++merged;
      sm100::tc_fence_after();
      const float2 with = merge[row];
      const float next = max_nan(m, with.x), base = max_nan(next, LOWEST);      // as in the blocks' loop
      const float a0 = ex2((m - base) * c2), a1 = ex2((with.x - base) * c2);
      l = l * a0 + with.y * a1;
      inv = 1.f / l;
      m = next;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t o1[16];
        sm100::tmem_ld_32x16(tmem_o + TMEM_COLS + q * 16, o1);
        sm100::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          o[q * 16 + i] = __float_as_uint(__uint_as_float(o[q * 16 + i]) * a0 + __uint_as_float(o1[i]) * a1);
      }
    }
    sm100::tc_fence_before();
    __syncwarp();
    if (lane == 0) {
      sm100::mbar_arrive(&sh->o_empty);
      if (merges) { sm100::mbar_arrive(&other_team->o_empty); sm100::mbar_arrive(&other_team->merge_empty); }
    }
    const int b = it.bh / p.H, h = it.bh - b * p.H;
    const size_t t = (size_t)it.qblk * BQ + row;
    __nv_bfloat16* out = p.out + ((size_t)b * p.T + t) * p.ld_out + h * D + half * 32;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[i] = pack_bf16(__float_as_uint(__uint_as_float(o[u * 8 + 2 * i]) * inv), __float_as_uint(__uint_as_float(o[u * 8 + 2 * i + 1]) * inv));
      *reinterpret_cast<uint4*>(out + u * 8) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (p.lse && half == 0) p.lse[(size_t)it.bh * p.T + t] = m * c2 * 0.6931471805599453f + __logf(l);
    if (tracer) stamp(p, r, it.qblk, 6);
  }
}

// SHARED: both teams of a CTA work on each of its items, half of the key blocks each (see attention_shares).  A template
// parameter: as an argument it cost the other form registers (8 x 16 x 1024 forward and backward 170 -> 174 us).
template <bool SHARED>
__global__ void __launch_bounds__(THREADS, 1)
attention_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];   // no static shared memory: the tiles start aligned
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* tiles = smem_raw + team() * SMEM_TILES;
  Shared* sh = (Shared*)(smem_raw + TEAMS * SMEM_TILES + team() * SMEM_SHARED);
  if (warp < 2 && sm100::elect_one()) {
    sm100::tma_prefetch_desc(&map_q);
    sm100::tma_prefetch_desc(&map_k);
    sm100::tma_prefetch_desc(&map_v);
    for (int s = 0; s < 2; ++s) {
      sm100::mbar_init(&sh->q_full[s], 1); sm100::mbar_init(&sh->q_empty[s], 1);
      sm100::mbar_init(&sh->k_full[s], 1); sm100::mbar_init(&sh->k_empty[s], 1);
      sm100::mbar_init(&sh->v_full[s], 1); sm100::mbar_init(&sh->v_empty[s], 1);
    }
    sm100::mbar_init(&sh->s_full, 1);
    sm100::mbar_init(&sh->s_empty, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->p_full, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->pv_done, 1);
    sm100::mbar_init(&sh->o_empty, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->merge_full, SOFTMAX_WARPS);
    sm100::mbar_init(&sh->merge_empty, SOFTMAX_WARPS);
    sh->error = 0;
    sm100::fence_barrier_init();
  }
  Shared* sh0 = (Shared*)(smem_raw + TEAMS * SMEM_TILES);
  if (warp == 2) {
    sm100::tmem_alloc(&sh0->tmem_base, TEAMS * TMEM_COLS);
    sm100::tmem_relinquish();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  if (threadIdx.x == 0) ((Shared*)((unsigned char*)sh0 + SMEM_SHARED))->tmem_base = sh0->tmem_base + TMEM_COLS;
  __syncthreads();

  wait_previous();
  // the swizzled tiles need a 1024-byte aligned base
  const bool fits = (sm100::smem_u32(tiles) & 1023u) == 0;
  if (!fits) {
    if (lane == 0) fail(sh, p, 9);
  } else if (warp < 4) {                                   // registers per four warps: 56 + 4 * 104 of the launch's 5 * 96
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp < 2) {
      if (sm100::elect_one()) producer<SHARED>(sh, tiles, p, &map_q, &map_k, &map_v);
    } else {
      if (sm100::elect_one()) mma_issuer<SHARED>(sh, tiles, p);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    float* xch = (float*)(smem_raw + TEAMS * (SMEM_TILES + SMEM_SHARED) + team() * XCH_BYTES);
    float2* merge = (float2*)(smem_raw + TEAMS * (SMEM_TILES + SMEM_SHARED + XCH_BYTES));
    Shared* other_team = (Shared*)(smem_raw + TEAMS * SMEM_TILES + (team() ^ 1) * SMEM_SHARED);
    softmax_rows<SHARED>(sh, other_team, xch, merge, p, warp & 3, ((warp - 4) >> 2) & 1, lane);
  }
  __syncwarp();
  sm100::tc_fence_before();
  __syncthreads();
  if (sh->error && warp < 2 && sm100::elect_one()) {
    const unsigned long long t0 = sm100::now_ns();
    while (sm100::now_ns() - t0 < 200000000ull) { __nanosleep(1000); }   // copies in flight land within microseconds
  }
  __syncthreads();
  if (warp == 2) {
    sm100::tc_fence_after();
    sm100::tmem_dealloc(sh0->tmem_base, TEAMS * TMEM_COLS);
  }
}

}  // namespace attn

static unsigned long long* g_attn_trace = nullptr;

// Time of the busiest unit (a team, or a CTA whose teams share) of a launch, in twentieths of a key block: its items in snake order,
// as Items deals them, and two blocks for each (Q and the first S before, the output or the merge after; one where a shared item is
// one block and has no merge).  A block of an item that is a team's own takes nine tenths of one that is shared.  One pass over
// the units per round, in runs of equal items.
static int attention_busiest(int items, int per_block, int q_blocks, int units, bool shared) {
  int load[1024] = {};
  for (int round = 0, t = 0; t < items; ++round) {
    const int end = std::min(items, t + units);
    int at = 0, blocks = q_blocks - t / per_block, run = per_block - t % per_block;
    for (; t < end; --blocks, run = per_block) {
      const int n = std::min(run, end - t), cost = shared ? (blocks + 1) / 2 * 20 + (blocks > 1 ? 40 : 20) : 18 * blocks + 40;
      int* l = load + ((round & 1) ? units - at - n : at);
      for (int k = 0; k < n; ++k) l[k] += cost;
      at += n;
      t += n;
    }
  }
  return *std::max_element(load, load + units);
}

// Whether the teams of a CTA share its items.  The launch takes as long as its busiest unit.  Sharing halves the longest item
// where there are few, and costs the fixed part twice where there are many; between one and three items per CTA it turns on
// how many of them the busiest one gets, which an average does not show.  Beyond that a team per item was faster throughout.
// Measured over 1 - 256 items of each length, lengths of 1 - 32 blocks, on 148 SMs (a team per item, shared, in us): 16 x 16 (heads
// x blocks) 30.4, 25.0; 37 x 8 18.7, 18.2; 64 x 3 10.2, 10.7; 52 x 4 11.7, 12.5; 27 x 13 27.4, 30.4; 20 x 20 39.9, 46.5; 128 x 8
// 47.3, 60.4.  The form taken is the faster one of both, or within 1.7 % of it, at each of those sizes.
static bool attention_shares(int per_block, int q_blocks, int grid) {      // per_block: items of each length, one to q_blocks
  const long long items = (long long)per_block * q_blocks;
  if (q_blocks < 2 || items > 4 * grid || attn::TEAMS * grid > 1024) return false;
  return attention_busiest((int)items, per_block, q_blocks, grid, true) < attention_busiest((int)items, per_block, q_blocks, attn::TEAMS * grid, false);
}

static int* attn_status_word(int** host_out = nullptr) {
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

// form: 0 a team per item, 1 the teams of a CTA share their items, -1 the rule's choice
static int attention_fwd(const void* q, const void* k, const void* v, int64_t ld_qkv, void* out, int64_t ld_out, float* lse,
                         int B, int T, int H, float scale, int form, void* stream) {
  if (B < 1 || H < 1 || T < 128 || T % 128) return fail(TMPI_ERR_UNSUPPORTED, "attention: T=%d must be a positive multiple of 128", T);
  if (ld_out % 8 || ((uintptr_t)out & 15)) return fail(TMPI_ERR_INVALID, "attention: the output must be 16-byte aligned with a pitch that is a multiple of 8");
  if ((int64_t)B * H * (T / 128) > 0x7fffffffLL) return fail(TMPI_ERR_INVALID, "attention: too many blocks");
  CUtensorMap mq, mk, mv;
  int st;
  const uint64_t rows = (uint64_t)B * T, cols = (uint64_t)H * attn::D;
  if ((st = make_tmap_bf16(&mq, q, rows, cols, (uint64_t)ld_qkv, 128))) return st;
  if ((st = make_tmap_bf16(&mk, k, rows, cols, (uint64_t)ld_qkv, 128))) return st;
  if ((st = make_tmap_bf16(&mv, v, rows, cols, (uint64_t)ld_qkv, 128))) return st;
  attn::Params p;
  p.B = B; p.T = T; p.H = H; p.q_blocks = T / attn::BQ;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.out = (__nv_bfloat16*)out; p.ld_out = (int)ld_out; p.lse = lse;
  p.status = attn_status_word();
  p.trace = g_attn_trace;
  p.items = B * H * p.q_blocks;
  // one CTA of two teams per SM, persistent; with fewer items than SMs each gets an SM of its own
  const int grid = std::min(p.items, gemm_sm_count());
  // a trace follows one team through an item; steep scales: see softmax_rows
  const bool shared = form < 0 ? !p.trace && p.scale_log2 <= 1.f && attention_shares(B * H, p.q_blocks, grid) : form != 0;
  const auto kernel = shared ? attn::attention_fwd_kernel<true> : attn::attention_fwd_kernel<false>;
  cudaError_t ae = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, attn::SMEM_BYTES);
  if (ae != cudaSuccess) return fail(TMPI_ERR_CUDA, "attention: shared memory attribute: %s", cudaGetErrorString(ae));
  cudaError_t e = launch_overlapped(kernel, grid, attn::THREADS, attn::SMEM_BYTES, (cudaStream_t)stream, mq, mk, mv, p);
  return e == cudaSuccess ? TMPI_OK : fail(TMPI_ERR_CUDA, "attention launch: %s", cudaGetErrorString(e));
}

extern "C" {

// out[b, t, h, :] = sum_s softmax_s(scale * q[b, t, h, :] . k[b, s, h, :], s <= t) v[b, s, h, :] for bf16 q, k, v given
// as [B * T, H * 64] matrices with a common row pitch of ld_qkv elements (for instance the three column blocks of a
// fused QKV projection); out is [B * T, ld_out]; lse (optional) is [B, H, T] fp32.  T must be a multiple of 128.
int tmpi_attention_fwd(const void* q, const void* k, const void* v, int64_t ld_qkv, void* out, int64_t ld_out, float* lse,
                       int B, int T, int H, float scale, void* stream) {
  return attention_fwd(q, k, v, ld_qkv, out, ld_out, lse, B, T, H, scale, -1, stream);
}

// The same in a given form (for tests and timing), and the form that tmpi_attention_fwd takes for scales of up to ln 2.
int tmpi_attention_fwd_form(const void* q, const void* k, const void* v, int64_t ld_qkv, void* out, int64_t ld_out, float* lse,
                            int B, int T, int H, float scale, int shared, void* stream) {
  return attention_fwd(q, k, v, ld_qkv, out, ld_out, lse, B, T, H, scale, shared != 0, stream);
}
int tmpi_attention_fwd_shares(int B, int T, int H) {
  const int64_t items = (int64_t)B * H * (T / attn::BQ);
  if (B < 1 || H < 1 || T < attn::BQ || items > 0x7fffffffLL) return 0;
  return attention_shares(B * H, T / attn::BQ, (int)std::min<int64_t>(items, gemm_sm_count()));
}

// Resident CTAs of the attention kernel per SM (1: a CTA holds two teams that overlap each other).
int tmpi_attention_ctas_per_sm(void) {
  int n = 0;
  cudaFuncSetAttribute(attn::attention_fwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn::SMEM_BYTES);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, attn::attention_fwd_kernel<false>, attn::THREADS, attn::SMEM_BYTES) != cudaSuccess) return -1;
  return n;
}

// Tuning aid: with a device buffer of (T / 128) * 16 64-bit words, team 0 of CTA 0 in every later launch (the last query block
// of the first batch and head) records the time of each phase of each key block of its first item (ns): 0 waits for S,
// 1 has S, 2 row maximum known, 3 P written, 4 P announced, 5 knows that P V is done, 6 the same (last block: output
// written); MMA thread: 8 waits to issue the next S, 9 next S issued, 10 has P, 11 has V, 12 P V issued.  nullptr
// switches it off.

void tmpi_attention_set_trace(void* device_buffer) { g_attn_trace = (unsigned long long*)device_buffer; }

// Non-zero after an attention CTA gave up on a bounded wait (3000 + the point where it happened); clears it.
int tmpi_attention_status(void) {
  int* host = nullptr;
  attn_status_word(&host);
  if (!host) return 0;
  int v = *(volatile int*)host;
  if (v) *(volatile int*)host = 0;
  return v;
}

}  // extern "C"
