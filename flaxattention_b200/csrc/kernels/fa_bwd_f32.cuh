// Flash-attention backward with fp32 inputs on the tensor cores (D = Dv = 64): the single pass of
// fa_bwd_tc.cuh (see there for the products and the reference citations) with every operand as three bf16
// parts, hi + mid + lo, which hold all the mantissa bits of an fp32 value; a product is the six bf16
// products of parts above 2^-25 of the largest, accumulated in fp32 (fa_fwd_tc.cuh describes the form).
// q, k, v and dO come as rows [hi | mid | lo] from a small kernel in front of this one, P and dS are split
// by the threads that compute them.  Heads with a value that has no parts are done over by fa_bwd_rerun_kernel.
//
// A pair is 128 kv rows x 64 query rows.  What shapes the kernel:
//   * Shared memory: the parts of K, V (96 KB), dS (48 KB) and three Q / dO tiles (72 KB).  Q and dO tiles pass
//     through a ring of three, dO(n), Q(n), dO(n+1), ..; product 3 frees dO(n) for Q(n+1), product 4 frees
//     Q(n) for dO(n+2).
//   * One warp issues all products, in the order 3(n) 2(n+1) 1(n+1) 4(n) 5(n): the scores of pair n+1 are
//     there when two products of pair n are still to run, and the element-wise work of n+1 runs under them.
//   * The tensor core adds into an fp32 accumulator without rounding to nearest, so dV, dK and dQ start from
//     zero for every pair and are added up elsewhere: dV and dK in the registers of one warpgroup (128
//     values per kv row), dQ by vector reductions to global memory.
//   * dQ = dS K has only 64 rows (M = 128 is the full rate): A is two parts of dS side by side along M,
//     [hi; mid] with lo, mid and hi of K, and [mid; lo] with hi of K, of which the lower half counts.
// Persistent, one CTA per SM, items handed out as in fa_bwd_tc.cuh.
//
// Warp roles (16 warps): 0-7 compute (thread = kv row, 32 query columns), 8-11 sums (dV, dK, dQ),
// 12 producer (pair lists, TMA loads), 13 MMA issuer and TMEM owner.
//
// TMEM columns: S^T 0-63, dP^T 64-127, P^T 128-223 (hi, mid, lo), dV 224-287, dK 288-351, dQ 352-415 and
// 416-479 ([mid; lo] . K hi).  Every mbarrier wait is bounded (see fa_sm100.cuh).
#pragma once
#include "fa_sm100.cuh"

struct FaBwdF32Params {
  FaParams p;
  FaTensorMap tq, tk, tv, tdo;  // the split tensors: 4-d maps (192, S, H, B), box 64 values x 64 rows (q, do) or 128 rows (k, v)
  const float* nlse2;           // [B, Hq, ceil(Sq/128)*128]: -lse * log2(e); -inf for rows without mass / beyond Sq
  const float* ndelta;          // same shape: -rowsum(O * dO); 0 beyond Sq
  int* work_counter;            // zero at launch
};

namespace fa_bf32 {

constexpr int DT = FA_DT_BF16;
constexpr int D = 64, BT = 128, BQ = 64, CW = 32;
constexpr int ATOM = 128 * 128;            // one part of a K, V or dS tile: 128 rows x 128 bytes
constexpr int QATOM = BQ * 128;            // one part of a Q or dO tile
constexpr int KV_BYTES = 3 * ATOM, Q_BYTES = 3 * QATOM;
constexpr int MAXPL = 512;                 // (head, q tile) pairs of one item
constexpr int MAXC = 256;                  // 128-row q tiles per head
constexpr int NT = 512;
constexpr int WARP_PRODUCER = 12, WARP_MMA = 13;
// Register split: 128 per thread at launch; the last warpgroup gives up 64 each, the compute warps take 8 each
// and the summing warpgroup, which holds 128 sums per thread, 48.
constexpr int REGS_COMPUTE = 136, REGS_SUMS = 176, REGS_OTHER = 64;
static_assert(256 * (REGS_COMPUTE - 128) + 128 * (REGS_SUMS - 128) <= 128 * (128 - REGS_OTHER), "setmaxnreg.inc would wait forever");

constexpr int OFF_K = 0, OFF_V = KV_BYTES, OFF_RING = 2 * KV_BYTES, OFF_DS = OFF_RING + 3 * Q_BYTES;
constexpr int OFF_ROW = OFF_DS + 3 * ATOM;                  // 3 x (nlse2[BQ], ndelta[BQ]), with the Q tile of the slot
constexpr int NBARS = 21;
constexpr int OFF_BAR = OFF_ROW + 3 * 2 * BQ * 4;
constexpr int OFF_MISC = OFF_BAR + NBARS * 8 + 8;           // tmem base, abort
constexpr int OFF_ITEM = OFF_MISC + 16;                     // int item[2][2]
constexpr int OFF_PAIR = OFF_ITEM + 16;                     // int pair[2][MAXPL]: q tile | mode << 16 | g << 20
constexpr int OFF_CLS = OFF_PAIR + 2 * MAXPL * 4;
constexpr int SMEM_BYTES = OFF_CLS + MAXC + 1024;
static_assert(SMEM_BYTES <= 227 * 1024 - 128, "shared memory");
static_assert(OFF_MISC % 16 == 0, "alignment");
constexpr int TMEM_COLS = 512;
constexpr int COL_S = 0, COL_DP = 64, COL_P = 128, COL_DV = 224, COL_DK = 288, COL_DQ = 352, COL_DQ2 = 416;

constexpr int BAR_KV = 0;                   // K and V of an item have landed
constexpr int BAR_FINAL = 1;                // the last product of an item is complete (K and V are free)
constexpr int BAR_FULL = 2, BAR_EMPTY = 5;  // [3] ring slots
constexpr int BAR_SFULL = 8;                // S^T and dP^T of a pair are in TMEM
constexpr int BAR_PREADY = 9;               // P^T in TMEM and dS^T in shared memory (256 arrivals)
constexpr int BAR_DSFREE = 10;              // products 4 and 5 of a pair are complete
constexpr int BAR_DVFULL = 11, BAR_DVFREE = 12, BAR_DKFULL = 13, BAR_DKFREE = 14, BAR_DQFULL = 15, BAR_DQFREE = 16;
constexpr int BAR_LISTFULL = 17, BAR_LISTFREE = 19;  // [2]
constexpr int LIST_CONSUMERS = 1 + 8 + 4;

__device__ __forceinline__ fa_u32 bar_addr(fa_u32 sb, int i) { return sb + OFF_BAR + i * 8; }
// parts of the two operands of the products kept, smallest first
__device__ constexpr int PA[6] = {1, 0, 2, 0, 1, 0}, PB[6] = {1, 2, 0, 1, 0, 0};

// The (query head, q tile) pairs of one item (as in fa_bwd_tc.cuh, two pairs per 128-row q tile).
__device__ __forceinline__ int build_pair_list(const FaParams& p, int hk, int b, int kt, int G, int n_ctiles,
                                               unsigned char* cl, int* pl, int lane) {
  const bool tables = p.t.kv_num != nullptr && p.t.q_num != nullptr;
  int w = 0;
  for (int g = 0; g < G; ++g) {
    if (!tables) {
      const int nq = (p.Sq + BQ - 1) / BQ, mode = FA_HAS_MASK_MOD ? 1 : 2;
      for (int e = lane; e < nq && w + e < MAXPL; e += 32) pl[w + e] = e | (mode << 16) | (g << 20);
      w += nq;
      continue;
    }
    const int h = hk * G + g;
    ((uint2*)cl)[lane] = make_uint2(0u, 0u);
    __syncwarp();
    const int bm = p.t.mB == 1 ? 0 : b, hm = p.t.mH == 1 ? 0 : h;
    const int kvblk = min(kt * BT / p.t.KVB, p.t.nKV - 1);
    const long long row = ((long long)bm * p.t.mH + hm) * p.t.nKV + kvblk;
    const int tpb = p.t.nQ == 1 ? n_ctiles : p.t.QB / 128;
    int num[2];
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const int* nump = which ? p.t.full_q_num : p.t.q_num;
      num[which] = nump != nullptr ? min(max(nump[row], 0), p.t.nQ) * tpb : 0;
    }
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const int* idxp = which ? p.t.full_q_idx : p.t.q_idx;
      for (int e = lane; e < num[which]; e += 32) {
        const int bi = e / tpb, ti = e - bi * tpb;
        const int t = min(max(idxp[row * p.t.nQ + bi], 0), p.t.nQ - 1) * tpb + ti;
        if (t < n_ctiles) cl[t] = (unsigned char)(which ? 2 : 1);
      }
      __syncwarp();
    }
    for (int t0 = 0; t0 < n_ctiles; t0 += 32) {
      const int t = t0 + lane;
      const int c = t < n_ctiles ? (int)cl[t] : 0;
      const int n_t = c == 0 ? 0 : ((2 * t + 1) * BQ < p.Sq ? 2 : 1);
      int inc = n_t;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      for (int v = 0; v < n_t; ++v)
        if (w + inc - n_t + v < MAXPL) pl[w + inc - n_t + v] = (t * 2 + v) | (c << 16) | (g << 20);
      w += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncwarp();
  }
  return min(w, MAXPL);
}

// 16 scores s and dp of kv row `kv`, query columns q0 .. q0+15 -> p (in s) and ds (in dp), fp32.  The operations
// and their order are those of fa_bwd.cuh.
__device__ __forceinline__ void elem16(float (&s)[16], float (&dp)[16], const float* nlse2, const float* ndelta, fa_u32 keep,
                                       int q0, int kv, int gb, int gh, float scale, float sc2) {
#pragma unroll
  for (int e = 0; e < 16; e += 4) {
    const float4 nl = *(const float4*)(nlse2 + e);
    const float4 nd = *(const float4*)(ndelta + e);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int qi = q0 | (e + u);
      const float nlu = u == 0 ? nl.x : (u == 1 ? nl.y : (u == 2 ? nl.z : nl.w));
      const float ndu = u == 0 ? nd.x : (u == 1 ? nd.y : (u == 2 ? nd.z : nd.w));
      float g = 1.f, x;
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_MUL_ONLY)
      g = fa_score_mul(0.f, gb, gh, qi, kv);
      x = fmaf(s[e + u], g * sc2, nlu);
#elif FA_HAS_SCORE_MOD
      g = fa_score_mod_grad(s[e + u] * scale, gb, gh, qi, kv);
      x = fmaf(fa_score_mod(s[e + u] * scale, gb, gh, qi, kv), FA_LOG2E, nlu);
#else
      x = fmaf(s[e + u], sc2, nlu);
#endif
      // (both are selected: the derivative of a score_mod may be infinite where the mask is false, and 0 times that is NaN)
      const bool in = (keep >> (e + u)) & 1u;
      const float pr = fa_ex2(x);
      s[e + u] = in ? pr : 0.f;
      dp[e + u] = in ? pr * (dp[e + u] + ndu) * g : 0.f;
    }
  }
}

}  // namespace fa_bf32

extern "C" __global__ void __launch_bounds__(fa_bf32::NT, 1) fa_bwd_f32_kernel(const __grid_constant__ FaBwdF32Params P) {
  using namespace fa_bf32;
  const FaParams& p = P.p;
  extern __shared__ unsigned char smem_raw[];
  if (fa_dynamic_smem_size() < (fa_u32)SMEM_BYTES || blockDim.x != NT) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicOr(p.status, FA_STATUS_BAD_LAUNCH);
    return;
  }
  FA_MOD_BUFS_INIT(p);
  const fa_u32 raw = fa_smem_u32(smem_raw);
  const fa_u32 sb = (raw + 1023u) & ~1023u;
  unsigned char* sm = smem_raw + (sb - raw);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.Hq / p.Hkv;
  const int n_ctiles = min((p.Sq + 127) / 128, MAXC);
  const int sq_pad = ((p.Sq + 127) / 128) * 128;
  const int n_items = p.Hkv * p.B * ((p.Skv + BT - 1) / BT);
  const int Gd = (int)gridDim.x, cta = (int)blockIdx.x;

  volatile int* misc = (volatile int*)(sm + OFF_MISC);
  int* pairs = (int*)(sm + OFF_PAIR);
  volatile int* item = (volatile int*)(sm + OFF_ITEM);

  if (tid == 0) {
    fa_mbar_init(bar_addr(sb, BAR_KV), 1);
    fa_mbar_init(bar_addr(sb, BAR_FINAL), 1);
    for (int s = 0; s < 3; ++s) {
      fa_mbar_init(bar_addr(sb, BAR_FULL + s), 1);
      fa_mbar_init(bar_addr(sb, BAR_EMPTY + s), 1);
    }
    fa_mbar_init(bar_addr(sb, BAR_SFULL), 1);
    fa_mbar_init(bar_addr(sb, BAR_PREADY), 256);
    fa_mbar_init(bar_addr(sb, BAR_DSFREE), 1);
    fa_mbar_init(bar_addr(sb, BAR_DVFULL), 1);
    fa_mbar_init(bar_addr(sb, BAR_DVFREE), 128);
    fa_mbar_init(bar_addr(sb, BAR_DKFULL), 1);
    fa_mbar_init(bar_addr(sb, BAR_DKFREE), 128);
    fa_mbar_init(bar_addr(sb, BAR_DQFULL), 1);
    fa_mbar_init(bar_addr(sb, BAR_DQFREE), 128);
    for (int i = 0; i < 2; ++i) {
      fa_mbar_init(bar_addr(sb, BAR_LISTFULL + i), 1);
      fa_mbar_init(bar_addr(sb, BAR_LISTFREE + i), LIST_CONSUMERS);
    }
    fa_mbar_init_fence();
    misc[1] = 0;
    fa_tma_prefetch_desc(&P.tk);
    fa_tma_prefetch_desc(&P.tv);
    fa_tma_prefetch_desc(&P.tq);
    fa_tma_prefetch_desc(&P.tdo);
  }
  if (warp == WARP_MMA) fa_tmem_alloc(sb + OFF_MISC, TMEM_COLS);
  fa_grid_wait();
  fa_tc_fence_before();
  __syncthreads();
  fa_tc_fence_after();
  const fa_u32 tmem = (fa_u32)misc[0];
  volatile int* abort_flag = misc + 1;
  const fa_u32 tmem_u = __shfl_sync(0xffffffffu, tmem, 0);

  if (warp >= 12) fa_setmaxnreg_dec<REGS_OTHER>();
  // Barrier phases: pair-indexed barriers count the pairs of the CTA across its items (gn), ring slots the tiles
  // (2 gn: dO, 2 gn + 1: Q), BAR_KV / BAR_FINAL the items that have pairs (kvc), the list barriers all items (itc).
  if (warp == WARP_PRODUCER) {
    // ================================ producer ================================================
    bool ok = true;
    int gn = 0, kvc = 0, idx = cta;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      if (itc >= 2) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFREE + lb), (fa_u32)(((itc >> 1) - 1) & 1), abort_flag);
      if (!ok) break;
      int* pl = pairs + lb * MAXPL;
      const int hk = idx % p.Hkv, b = (idx / p.Hkv) % p.B, kt = idx / (p.Hkv * p.B);
      int np = -1;
      if (idx < n_items) np = build_pair_list(p, hk, b, kt, G, n_ctiles, sm + OFF_CLS, pl, lane);
      if (lane == 0) {
        item[2 * lb] = idx;
        item[2 * lb + 1] = np;
      }
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFULL + lb));
      if (np < 0) break;
      int next = 0;
      if (lane == 0) {
        next = Gd + atomicAdd(P.work_counter, 1);
        const int n0 = kt * BT;
        // K and V are free when the last product of the previous item is complete; the tiles of this item's
        // first pair have their ring slots earlier and go first
        for (int n = 0; n < np && ok; ++n, ++gn) {
          const int pr = pl[n];
          const int m0 = (pr & 0xffff) * BQ, h = hk * G + (pr >> 20);
          for (int which = 0; which < 2 && ok; ++which) {
            const int t = 2 * gn + which, s = t % 3;
            if (t >= 3) ok = fa_mbar_wait(bar_addr(sb, BAR_EMPTY + s), (fa_u32)((t / 3 - 1) & 1), abort_flag);
            if (!ok) break;
            const fa_u32 full = bar_addr(sb, BAR_FULL + s);
            fa_mbar_expect_tx(full, Q_BYTES + (which ? 2 * BQ * 4 : 0));
            for (int a = 0; a < 3; ++a)
              fa_tma_load_4d(sb + OFF_RING + s * Q_BYTES + a * QATOM, which ? &P.tq : &P.tdo, full, a * 64, m0, h, b);
            if (which) {
              const long long rbase = ((long long)b * p.Hq + h) * sq_pad + m0;
              fa_bulk_load(sb + OFF_ROW + s * 2 * BQ * 4, P.nlse2 + rbase, BQ * 4, full);
              fa_bulk_load(sb + OFF_ROW + s * 2 * BQ * 4 + BQ * 4, P.ndelta + rbase, BQ * 4, full);
            }
            if (n == 0 && which == 0) {
              if (kvc > 0) ok = fa_mbar_wait(bar_addr(sb, BAR_FINAL), (fa_u32)((kvc - 1) & 1), abort_flag);
              if (!ok) break;
              fa_mbar_expect_tx(bar_addr(sb, BAR_KV), 2 * KV_BYTES);
              for (int a = 0; a < 3; ++a) {
                fa_tma_load_4d(sb + OFF_K + a * ATOM, &P.tk, bar_addr(sb, BAR_KV), a * 64, n0, hk, b);
                fa_tma_load_4d(sb + OFF_V + a * ATOM, &P.tv, bar_addr(sb, BAR_KV), a * 64, n0, hk, b);
              }
            }
          }
        }
      }
      if (np > 0) ++kvc;
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      gn = __shfl_sync(0xffffffffu, gn, 0);
      idx = __shfl_sync(0xffffffffu, next, 0);
    }
  } else if (warp == WARP_MMA) {
    // ================================ MMA issuer ===============================================
    const bool leader = fa_elect_one();
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    constexpr fa_u32 IDESC_KK = fa_idesc(DT, 128, BQ, 0, 0);  // A, B K-major
    constexpr fa_u32 IDESC_KN = fa_idesc(DT, 128, D, 0, 1);   // A K-major (TMEM or smem), B MN-major
    constexpr fa_u32 IDESC_NN = fa_idesc(DT, 128, D, 1, 1);   // A, B MN-major
    const fa_u32 loK = fa_desc_lo(sb + OFF_K, 16), loV = fa_desc_lo(sb + OFF_V, 16), loDS = fa_desc_lo(sb + OFF_DS, 16);
    const fa_u32 loDS_mn = fa_desc_lo(sb + OFF_DS, ATOM), loK_mn = fa_desc_lo(sb + OFF_K, ATOM);
    // d = A B^T over 64 values: A from smem at `a` (parts ATOM apart), B at `b` (parts QATOM apart), both K-major
    auto product_kk = [&](int col, fa_u32 a, fa_u32 b) {
#pragma unroll
      for (int pr = 0; pr < 6; ++pr)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (leader)
            fa_mma_ss(tmem_u + col, fa_desc_make(a + ((PA[pr] * ATOM + kk * 32) >> 4), HI), fa_desc_make(b + ((PB[pr] * QATOM + kk * 32) >> 4), HI),
                      IDESC_KK, pr > 0 || kk > 0);
    };
    auto tile_lo = [&](int t) { return fa_desc_lo(sb + OFF_RING + (t % 3) * Q_BYTES, 16); };
    auto wait_tile = [&](int t) { return fa_mbar_wait_each(bar_addr(sb, BAR_FULL + t % 3), (fa_u32)((t / 3) & 1), abort_flag); };
    bool ok = true;
    int gn = 0, kvc = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_each(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int np = __shfl_sync(0xffffffffu, item[2 * lb + 1], 0);
      __syncwarp();
      if (leader) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
      if (np < 0) break;
      if (np == 0) continue;
      ok = fa_mbar_wait_each(bar_addr(sb, BAR_KV), (fa_u32)(kvc & 1), abort_flag);
      // the scores of an item's first pair (those of the later ones are issued a pair ahead)
      if (ok) ok = wait_tile(2 * gn) && wait_tile(2 * gn + 1);
      if (!ok) break;
      fa_tc_fence_after();
      product_kk(COL_DP, loV, tile_lo(2 * gn));
      product_kk(COL_S, loK, tile_lo(2 * gn + 1));
      if (leader) fa_mma_commit(bar_addr(sb, BAR_SFULL));
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const fa_u32 prev = (fa_u32)((gn - 1) & 1);
        ok = fa_mbar_wait_each(bar_addr(sb, BAR_PREADY), (fa_u32)(gn & 1), abort_flag);
        if (ok && gn > 0) ok = fa_mbar_wait_each(bar_addr(sb, BAR_DVFREE), prev, abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        const fa_u32 loDO = tile_lo(2 * gn), loQ = tile_lo(2 * gn + 1);
        // 3. dV = P^T dO   (A from TMEM)
#pragma unroll
        for (int pr = 0; pr < 6; ++pr)
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk)
            if (leader)
              fa_mma_ts(tmem_u + COL_DV, tmem_u + COL_P + PA[pr] * 32 + kk * 8, fa_desc_make(loDO + ((PB[pr] * QATOM) >> 4) + kk * 128, HI),
                        IDESC_KN, pr > 0 || kk > 0);
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_EMPTY + (2 * gn) % 3));
          fa_mma_commit(bar_addr(sb, BAR_DVFULL));
        }
        if (n + 1 < np) {
          // 2. and 1. of the next pair (the compute warps have read this pair's scores: PREADY)
          ok = wait_tile(2 * gn + 2);
          if (!ok) break;
          fa_tc_fence_after();
          product_kk(COL_DP, loV, tile_lo(2 * gn + 2));
          ok = wait_tile(2 * gn + 3);
          if (!ok) break;
          fa_tc_fence_after();
          product_kk(COL_S, loK, tile_lo(2 * gn + 3));
          if (leader) fa_mma_commit(bar_addr(sb, BAR_SFULL));
        }
        // 4. dK = dS^T Q
        if (gn > 0) ok = fa_mbar_wait_each(bar_addr(sb, BAR_DKFREE), prev, abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
#pragma unroll
        for (int pr = 0; pr < 6; ++pr)
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk)
            if (leader)
              fa_mma_ss(tmem_u + COL_DK, fa_desc_make(loDS + ((PA[pr] * ATOM + kk * 32) >> 4), HI), fa_desc_make(loQ + ((PB[pr] * QATOM) >> 4) + kk * 128, HI),
                        IDESC_KN, pr > 0 || kk > 0);
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_EMPTY + (2 * gn + 1) % 3));
          fa_mma_commit(bar_addr(sb, BAR_DKFULL));
        }
        // 5. dQ = dS K: [hi; mid] with the parts of K, lo first, and [mid; lo] with hi of K
        if (gn > 0) ok = fa_mbar_wait_each(bar_addr(sb, BAR_DQFREE), prev, abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
#pragma unroll
        for (int pr = 0; pr < 4; ++pr)
#pragma unroll
          for (int kk = 0; kk < BT / 16; ++kk) {
            const int kpart = pr < 3 ? 2 - pr : 0;
            if (leader)
              fa_mma_ss(tmem_u + (pr < 3 ? COL_DQ : COL_DQ2), fa_desc_make(loDS_mn + (pr < 3 ? 0 : ATOM >> 4) + kk * 128, HI),
                        fa_desc_make(loK_mn + ((kpart * ATOM) >> 4) + kk * 128, HI), IDESC_NN, (pr > 0 && pr < 3) || kk > 0);
          }
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_DSFREE));
          fa_mma_commit(bar_addr(sb, BAR_DQFULL));
          if (n + 1 == np) fa_mma_commit(bar_addr(sb, BAR_FINAL));
        }
      }
      ++kvc;
    }
  } else if (warp < 8) {
    // ================================ compute warps ============================================
    fa_setmaxnreg_inc<REGS_COMPUTE>();
    const int half = warp >> 2;               // query columns 32 * half .. + 31 of the pair
    const int lane_base = (warp & 3) * 32;
    const int r = lane_base + lane;           // kv row inside the tile
    const fa_u32 t_row = tmem + ((fa_u32)lane_base << 16);
    const float sc2 = p.scale * FA_LOG2E;
    const bool bits = p.t.mask_bits_t != nullptr && (p.t.mask_hold == nullptr || *p.t.mask_hold != 0);
    bool ok = true;
    int gn = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int idx = item[2 * lb], np = item[2 * lb + 1];
      if (np < 0) break;
      const int* pl = pairs + lb * MAXPL;
      const int hk = idx % p.Hkv, b = (idx / p.Hkv) % p.B, n0 = (idx / (p.Hkv * p.B)) * BT;
      const int gb = b + p.b_off;
      const int kv = n0 + r;
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int s = (2 * gn + 1) % 3;
        const int pr = pl[n];
        const int q0 = (pr & 0xffff) * BQ + half * CW, mode = (pr >> 16) & 0xf, h = hk * G + (pr >> 20), gh = h + p.h_off;
        // which of this thread's columns count: bit e is query q0 + e
        fa_u32 keep = kv < p.Skv ? 0xffffffffu : 0u;
#if FA_HAS_MASK_MOD
        if (mode == 1 && kv < p.Skv) {
          if (bits) {
            // (the words of a row cover whole 128-query tiles of at least Sq queries)
            const long long e = (long long)(p.t.mask_B == 1 ? 0 : b) * p.t.mask_H + (p.t.mask_H == 1 ? 0 : h);
            keep = p.t.mask_bits_t[(e * p.t.mask_t_rows + kv) * p.t.mask_t_stride + (q0 >> 5)];
          } else {
            keep = 0u;
#pragma unroll 4
            for (int e = 0; e < CW; ++e) keep |= (fa_mask_mod(gb, gh, q0 + e, kv) ? 1u : 0u) << e;
          }
        }
#endif
        // (a score_mod may not be finite beyond Sq, and there the zero rows of Q and dO do not help)
        const int left = p.Sq - q0;
        if (left < CW) keep &= left <= 0 ? 0u : (1u << left) - 1u;
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_SFULL), (fa_u32)(gn & 1), abort_flag);
        if (ok) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_FULL + s), (fa_u32)(((2 * gn + 1) / 3) & 1), abort_flag);  // (the row scalars)
        if (!ok) break;
        fa_tc_fence_after();
        const float* rowp = (const float*)(sm + OFF_ROW + s * 2 * BQ * 4) + half * CW;
        float s0[16], d0[16], s1[16], d1[16];
        fa_tmem_ld16(t_row + COL_S + half * CW, s0);
        fa_tmem_ld16(t_row + COL_DP + half * CW, d0);
        fa_tmem_wait_ld();
        fa_tmem_ld16(t_row + COL_S + half * CW + 16, s1);
        fa_tmem_ld16(t_row + COL_DP + half * CW + 16, d1);
        // P^T goes to TMEM at once: product 3 of the last pair, its last reader, was issued before this pair's scores
        fa_u32 hi[8], mid[8], lo[8];
#define FA_STEP(SC, DC, C)                                                                                                    \
  elem16(SC, DC, rowp + (C), rowp + BQ + (C), keep >> (C), q0 + (C), kv, gb, gh, p.scale, sc2);                               \
  _Pragma("unroll") for (int e = 0; e < 8; ++e) fa_split3(fa_f2(SC[2 * e], SC[2 * e + 1]), hi[e], mid[e], lo[e]);             \
  fa_tmem_st8(t_row + COL_P + half * 16 + (C) / 2, hi);                                                                       \
  fa_tmem_st8(t_row + COL_P + 32 + half * 16 + (C) / 2, mid);                                                                 \
  fa_tmem_st8(t_row + COL_P + 64 + half * 16 + (C) / 2, lo);
        FA_STEP(s0, d0, 0)
        fa_tmem_wait_ld();
        FA_STEP(s1, d1, 16)
#undef FA_STEP
        // products 4 and 5 of the last pair must be done with dS^T
        if (gn > 0) {
          ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DSFREE), (fa_u32)((gn - 1) & 1), abort_flag);
          if (!ok) break;
        }
#define FA_STORE(DC, C)                                                                                                       \
  _Pragma("unroll") for (int e = 0; e < 8; ++e) fa_split3(fa_f2(DC[2 * e], DC[2 * e + 1]), hi[e], mid[e], lo[e]);             \
  _Pragma("unroll") for (int e = 0; e < 8; e += 4) {                                                                          \
    unsigned char* at = sm + OFF_DS + r * 128 + (((half * 4 + (C) / 8 + e / 4) ^ (r & 7)) * 16);                              \
    *(uint4*)at = make_uint4(hi[e], hi[e + 1], hi[e + 2], hi[e + 3]);                                                         \
    *(uint4*)(at + ATOM) = make_uint4(mid[e], mid[e + 1], mid[e + 2], mid[e + 3]);                                            \
    *(uint4*)(at + 2 * ATOM) = make_uint4(lo[e], lo[e + 1], lo[e + 2], lo[e + 3]);                                            \
  }
        FA_STORE(d0, 0)
        FA_STORE(d1, 16)
#undef FA_STORE
        fa_tmem_wait_st();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_PREADY));
      }
      if (!ok) break;
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
    }
  } else if (warp < 12) {
    // ================================ sums: dV and dK in registers, dQ to global memory =========
    fa_setmaxnreg_inc<REGS_SUMS>();
    const int lane_base = (warp & 3) * 32;
    const int r = lane_base + lane;  // kv row (dV, dK); for dQ the query row r & 63, upper or lower half of the stacked product
    const fa_u32 t_lane = tmem + ((fa_u32)lane_base << 16);
    bool ok = true;
    int gn = 0;
    float dv[D], dk[D];
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int idx = item[2 * lb], np = item[2 * lb + 1];
      if (np < 0) break;
      const int* pl = pairs + lb * MAXPL;
      const int hk = idx % p.Hkv, b = (idx / p.Hkv) % p.B, n0 = (idx / (p.Hkv * p.B)) * BT;
#pragma unroll
      for (int e = 0; e < D; ++e) dv[e] = dk[e] = 0.f;
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int pr = pl[n];
        float a[16];
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DVFULL), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
          fa_tmem_ld16(t_lane + COL_DV + 16 * c, a);
          fa_tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) dv[16 * c + e] += a[e];
        }
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_DVFREE));
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DKFULL), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
          fa_tmem_ld16(t_lane + COL_DK + 16 * c, a);
          fa_tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) dk[16 * c + e] += a[e];
        }
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_DKFREE));
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DQFULL), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        const int q = (pr & 0xffff) * BQ + (r & 63), h = hk * G + (pr >> 20);
        float* dq = (float*)p.dq.ptr + (long long)b * p.dq.sb + (long long)h * p.dq.sh + (long long)q * p.dq.ss;
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
          fa_tmem_ld16(t_lane + COL_DQ + 16 * c, a);
          if (warp >= 10) {  // lanes 64-127: mid . K, and lo . hi from the second product
            float y[16];
            fa_tmem_ld16(t_lane + COL_DQ2 + 16 * c, y);
            fa_tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) a[e] += y[e];
          } else {
            fa_tmem_wait_ld();
          }
          if (q < p.Sq) {
#pragma unroll
            for (int e = 0; e < 16; e += 4)
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dq + 16 * c + e), "f"(a[e] * p.scale), "f"(a[e + 1] * p.scale),
                           "f"(a[e + 2] * p.scale), "f"(a[e + 3] * p.scale)
                           : "memory");
          }
        }
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_DQFREE));
      }
      if (!ok) break;
      const int kv = n0 + r;
      if (kv < p.Skv) {
        float* gk = (float*)p.dk.ptr + (long long)b * p.dk.sb + (long long)hk * p.dk.sh + (long long)kv * p.dk.ss;
        float* gv = (float*)p.dv.ptr + (long long)b * p.dv.sb + (long long)hk * p.dv.sh + (long long)kv * p.dv.ss;
#pragma unroll
        for (int e = 0; e < D; e += 4) {
          *(float4*)(gk + e) = make_float4(dk[e] * p.scale, dk[e + 1] * p.scale, dk[e + 2] * p.scale, dk[e + 3] * p.scale);
          *(float4*)(gv + e) = make_float4(dv[e], dv[e + 1], dv[e + 2], dv[e + 3]);
        }
      }
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
    }
  }

  // ---- teardown ------------------------------------------------------------------------------
  fa_tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    fa_tc_fence_after();
    fa_tmem_dealloc(tmem, TMEM_COLS);
  }
  if (tid == 0 && *abort_flag != 0 && p.status != nullptr) atomicOr(p.status, FA_STATUS_WAIT_TIMEOUT);
}
