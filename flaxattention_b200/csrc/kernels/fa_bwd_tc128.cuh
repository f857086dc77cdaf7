// Flash-attention backward for sm_100a on the 5th-generation tensor cores, fp16 / bf16, D = Dv = 128: the single pass of
// fa_bwd_tc.cuh (see there for the products, the items and the reference citations) over pairs of 128 kv x 128 q rows.
//
// TMEM (512 columns) holds two 128-column accumulators (dK, dV), so the tiles of a pair share the other half:
//   S^T 0-127, over it P^T (16 bit; the compute warps write it where they have read the scores);
//   dP^T 128-255, over it dS^T (16 bit) in the same way, and over that dQ;  dV 256-383;  dK 384-511.
// One warp issues all products, in the order  S(n+1)  dK(n)  dQ(n)  dP(n+1)  dV(n+1): S(n+1) runs while the compute
// warps turn dP(n) into dS(n), dK(n) and dQ(n) while they compute P(n+1), dV(n+1) and S(n+2) while they turn
// dP(n+1) into dS(n+1).  The order itself says when a buffer is free: S^T(n+1) comes behind dV(n), the last reader
// of P^T(n), dQ(n) behind dK(n), which reads dS^T(n) from TMEM, and dP^T(n+1) behind both, so dP^T(n+1) in TMEM also means
// that the one dS^T buffer in shared memory may be written.  dP^T(n+1) alone waits for somebody else: the drain warps, which
// take dQ(n) out.
//
// Why this shape: an instruction with N = 128 reads 8 KB of operands for 64 clocks of math, one with N = 64 6 KB for 32,
// and shared memory delivers 128 bytes a clock: per 128 x 128 scores the five products read 256 KB (dV and dK take their A
// operand from TMEM) where pairs of 64 query rows read 384, and a pair has the same number of hand-overs between
// the roles for twice the work.  Against pairs of 64 query rows (kernel alone, us, both from one box): dense B4 H8 S4096
// 666 -> 582, attention sink B4 H16 S8192 865 -> 799, causal B2 H8 S4096 199 -> 173, causal + ALiBi B4 H16 S2048 234 -> 218.  Few rows that
// end early in a tile lose (B2 H4 S192, a pass: 17.0 -> 18.1): their last pair has 128 rows all the same.
#pragma once
#include "fa_bwd_items.cuh"

namespace fa_b128 {

constexpr int DT = FA_DTYPE;
constexpr int D = 128;
constexpr int BT = 128, BQ = 128;          // kv rows, q rows of a pair
constexpr int CW = BQ / 2;                 // q columns of one compute thread
constexpr int ATOM_BYTES = 128 * 128;      // 128 rows x 128 bytes (64 values)
constexpr int TILE_BYTES = 2 * ATOM_BYTES; // a K, V, Q, dO or dS^T tile
constexpr int NQS = 2;                     // Q tiles in flight; dO has one: it is read last by dV(n) and again by dP(n+1), three products later
constexpr int MAXPL = 1024;                // (head, q tile) pairs of one item (two such lists fit in shared memory)
constexpr int MAXC = 256;                  // q tiles per head (Sq <= 32768)
constexpr int NT = 512;
constexpr int WARP_PRODUCER = 12, WARP_MMA = 13;
// Register split (setmaxnreg), 128 per thread at launch: a drain thread holds a whole row of dQ (128 values), so that its
// TMEM columns are free after one round of loads; a compute thread the 64 probabilities between its two halves.
constexpr int REGS_COMPUTE = 136, REGS_DRAIN = 152, REGS_OTHER = 88;
static_assert(256 * (REGS_COMPUTE - 128) + 128 * (REGS_DRAIN - 128) <= 128 * (128 - REGS_OTHER), "setmaxnreg.inc would wait forever");

// shared memory map (from a 1024-byte aligned base)
constexpr int OFF_K = 0;
constexpr int OFF_V = OFF_K + TILE_BYTES;
constexpr int OFF_Q = OFF_V + TILE_BYTES;                   // NQS tiles
constexpr int OFF_DO = OFF_Q + NQS * TILE_BYTES;
constexpr int OFF_DS = OFF_DO + TILE_BYTES;                 // dS^T
constexpr int OFF_ST = OFF_DS + TILE_BYTES;                 // staging, 4 KB of each drain warp for dQ, together for dK / dV (64 columns at a time)
constexpr int OFF_ROW = OFF_ST + ATOM_BYTES;                // NQS x (nlse2[BQ], ndelta[BQ]) floats
constexpr int OFF_BAR = OFF_ROW + NQS * 2 * BQ * 4;
constexpr int NBARS = 22;
constexpr int OFF_MISC = OFF_BAR + NBARS * 8;               // tmem base, abort, -, drain flag
constexpr int OFF_ITEM = OFF_MISC + 16;                     // int item[2][4]: kv head, batch, kv tile, pairs (-1: no more work)
constexpr int OFF_PAIR = OFF_ITEM + 32;                     // int pair[2][MAXPL]: q tile | mode << 16 | g << 20
constexpr int OFF_CLS = OFF_PAIR + 2 * MAXPL * 4;           // unsigned cls[2][MAXC / 32] (scratch of the list builder)
constexpr int SMEM_BYTES = OFF_CLS + 2 * MAXC / 8 + 1024;
// (the pointers of up to eight captured buffers are static shared memory beside this)
static_assert(SMEM_BYTES + 8 * 8 <= 227 * 1024, "shared memory");
static_assert(OFF_MISC % 16 == 0, "alignment");
constexpr int TMEM_COLS = 512;
constexpr int COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 384;

constexpr int BAR_K = 0, BAR_V = 1;             // K / V of an item have landed
constexpr int BAR_KFREE = 2, BAR_VFREE = 3;     // the last product that reads K / V of an item is complete
constexpr int BAR_QFULL = 4, BAR_QEMPTY = 4 + NQS;       // [NQS] Q tile and row scalars
constexpr int BAR_DOFULL = 4 + 2 * NQS, BAR_DOEMPTY = BAR_DOFULL + 1;
constexpr int BAR_SFULL = BAR_DOFULL + 2;       // S^T of a pair is in TMEM
constexpr int BAR_PREADY = BAR_SFULL + 1;       // P^T is (256 arrivals)
constexpr int BAR_DPFULL = BAR_SFULL + 2;       // dP^T of a pair is in TMEM
constexpr int BAR_DSREADY = BAR_SFULL + 3;      // dS^T is in shared memory and TMEM, dP^T has been read (256 arrivals)
constexpr int BAR_DQFULL = BAR_SFULL + 4;       // dQ of a pair is in TMEM
constexpr int BAR_DQFREE = BAR_SFULL + 5;       // the drain warps hold it in registers (128 arrivals)
constexpr int BAR_FINAL = BAR_SFULL + 6;        // dK and dV of an item are complete
constexpr int BAR_DKVFREE = BAR_SFULL + 7;      // the drain warps have read them out of TMEM (128 arrivals)
constexpr int BAR_LISTFULL = BAR_SFULL + 8;     // [2] the producer has published an item and its pair list
constexpr int BAR_LISTFREE = BAR_SFULL + 10;    // [2] the consumers of a list are done with it
static_assert(BAR_LISTFREE + 2 <= NBARS, "barriers");
constexpr int LIST_CONSUMERS = 1 + 8 + 4;       // MMA issuer, compute warps, drain warps (one arrival each)

__device__ __forceinline__ fa_u32 bar_addr(fa_u32 sb, int i) { return sb + OFF_BAR + i * 8; }

// First half of the element-wise work on 16 columns of a thread's row: scores (raw) of kv row `kv`, q columns q0 .. q0+15
// -> P^T packed to 16 bits and pg = p * (derivative of the score_mod), what dS^T needs of them.  q0 is a multiple of 16
// (the compiler can see that from how the caller builds it).  nlse2 points at the row scalar of column q0.  Bit e of
// `keep` is the mask of column e, looked at if `masked`: as a select per element, which is faster here than masking the packed
// words as at head dim 64 (causal + ALiBi B4 H16 S2048 206 against 224 us, attention sink 815 / 823).  Both the probability and pg
// are selected, unless the tracer knows the derivative of the score_mod to be finite everywhere (FA_SCORE_GRAD_FINITE): it may be
// infinite where the mask is false, and 0 times that is NaN (the second select: causal + ALiBi B8 H8 S2048, with the conversion of
// dQ, 245 -> 254 us).
__device__ __forceinline__ void p_chunk(const float (&s)[16], const float* nlse2, fa_u32 (&pp)[8], float* pg, bool masked, fa_u32 keep,
                                        int q0, int kv, int gb, int gh, float scale, float sc2) {
#if !FA_HAS_SCORE_MOD || defined(FA_SCORE_AFFINE)
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_LINEAR_Q)
  // (a bias linear in q under a multiplier that does not read it: see fa_bwd_tc.cuh)
  const float lin_g = fa_score_mul(0.f, gb, gh, q0, kv);
  const fa_u64 lin_g2 = fa_f2(lin_g, lin_g), lin_gs2 = fa_f2(lin_g * sc2, lin_g * sc2);
  const float lin_base = fa_score_add2(0.f, gb, gh, q0, kv), lin_dq = fa_score_add2_dq(0.f, gb, gh, q0, kv);
  const fa_u64 lin_od[4] = {fa_f2(0.f, lin_dq), fa_f2(2.f * lin_dq, 3.f * lin_dq), fa_f2(4.f * lin_dq, 5.f * lin_dq), fa_f2(6.f * lin_dq, 7.f * lin_dq)};
  float at8 = lin_base;
#endif
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    const float2 nl = *(const float2*)(nlse2 + e);
    const fa_u64 nl2 = fa_f2(nl.x, nl.y);
    float s0 = s[e], s1 = s[e + 1];
#if FA_ROUND_SCORES
    fa_round2<DT>(s0, s1);
#endif
    const fa_u64 s2 = fa_f2(s0, s1);
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_LINEAR_Q)
    [[maybe_unused]] const fa_u64 g2 = lin_g2;
    if (e == 8) at8 = fmaf(8.f, lin_dq, lin_base);
    const fa_u64 x2 = fa_fma2(s2, lin_gs2, fa_add2(fa_add2(fa_f2(at8, at8), nl2), lin_od[(e % 8) / 2]));
#elif FA_HAS_SCORE_MOD
    const int qi0 = q0 | e, qi1 = q0 | (e + 1);
    const fa_u64 g2 = fa_f2(fa_score_mul(0.f, gb, gh, qi0, kv), fa_score_mul(0.f, gb, gh, qi1, kv));
    const fa_u64 b2 = fa_add2(fa_f2(fa_score_add2(0.f, gb, gh, qi0, kv), fa_score_add2(0.f, gb, gh, qi1, kv)), nl2);
    const fa_u64 x2 = fa_fma2(s2, fa_mul2(g2, fa_f2(sc2, sc2)), b2);
#else
    const fa_u64 x2 = fa_fma2(s2, fa_f2(sc2, sc2), nl2);
#endif
    float x0, x1;
    fa_f2_unpack(x2, x0, x1);
    float p0 = fa_ex2(x0), p1 = fa_ex2(x1);
#if FA_HAS_MASK_MOD || FA_BWD_CLEAR_BEYOND
    if (masked) {
      p0 = (keep >> e) & 1u ? p0 : 0.f;
      p1 = (keep >> (e + 1)) & 1u ? p1 : 0.f;
    }
#endif
    pp[e / 2] = fa_pack2<DT>(p0, p1);
#if FA_HAS_SCORE_MOD && !defined(FA_SCORE_MUL_ONE)
    fa_f2_unpack(fa_mul2(fa_f2(p0, p1), g2), pg[e], pg[e + 1]);
#if (FA_HAS_MASK_MOD || FA_BWD_CLEAR_BEYOND) && !defined(FA_SCORE_GRAD_FINITE)
    if (masked) {
      pg[e] = (keep >> e) & 1u ? pg[e] : 0.f;
      pg[e + 1] = (keep >> (e + 1)) & 1u ? pg[e + 1] : 0.f;
    }
#endif
#else
    pg[e] = p0;
    pg[e + 1] = p1;
#endif
  }
#else
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    const float2 nl = *(const float2*)(nlse2 + e);
    float pv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float nlu = u == 0 ? nl.x : nl.y;
      float x = s[e + u];
#if FA_ROUND_SCORES
      {
        float dummy = 0.f;
        fa_round2<DT>(x, dummy);
      }
#endif
      const float g = fa_score_mod_grad(x * scale, gb, gh, q0 | (e + u), kv);
      x = fa_score_mod(x * scale, gb, gh, q0 | (e + u), kv) * FA_LOG2E + nlu;
      float pr = fa_ex2(x);
      pg[e + u] = pr * g;
#if FA_HAS_MASK_MOD || FA_BWD_CLEAR_BEYOND
      if (masked && !((keep >> (e + u)) & 1u)) pr = pg[e + u] = 0.f;
#endif
      pv[u] = pr;
    }
    pp[e / 2] = fa_pack2<DT>(pv[0], pv[1]);
  }
#endif
}

// Second half: dS^T = pg (dP^T - delta), packed to 16 bits.  ndelta points at the row scalar of the first column.
__device__ __forceinline__ void ds_chunk(const float (&dp)[16], const float* ndelta, const float* pg, fa_u32 (&ds)[8]) {
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    const float2 nd = *(const float2*)(ndelta + e);
    float d0, d1;
    fa_f2_unpack(fa_mul2(fa_f2(pg[e], pg[e + 1]), fa_add2(fa_f2(dp[e], dp[e + 1]), fa_f2(nd.x, nd.y))), d0, d1);
    ds[e / 2] = fa_pack2<DT>(d0, d1);
  }
}

}  // namespace fa_b128

extern "C" __global__ void __launch_bounds__(fa_b128::NT, 1) fa_bwd_tc_kernel(const __grid_constant__ FaBwdTcParams P) {
  using namespace fa_b128;
  using namespace fa_bwd_items;
  const FaParams& p = P.p;
  extern __shared__ unsigned char smem_raw[];
  // a launch that does not fit the shared-memory map above (a host library built for another
  // version of this file) is refused before anything is written
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
  const int n_qtiles = min((p.Sq + 127) / 128, MAXC);
  const int sq_pad = ((p.Sq + 127) / 128) * 128;
  const int n_kvt = (p.Skv + BT - 1) / BT;
  const int n_items = p.Hkv * p.B * n_kvt;
  const int Gd = (int)gridDim.x, cta = (int)blockIdx.x;

  volatile int* misc = (volatile int*)(sm + OFF_MISC);  // [0] tmem base, [1] abort, [2] unused, [3] drain warps leave
  int* pairs = (int*)(sm + OFF_PAIR);                   // two lists of MAXPL pairs
  volatile int* item = (volatile int*)(sm + OFF_ITEM);  // per list: kv head, batch, kv tile, pairs

  // ---- set-up --------------------------------------------------------------------------------
  if (tid == 0) {
    for (int i = 0; i < NBARS; ++i) {
      const int count = (i == BAR_PREADY || i == BAR_DSREADY) ? 256
                        : (i == BAR_DQFREE || i == BAR_DKVFREE) ? 128
                        : (i == BAR_LISTFREE || i == BAR_LISTFREE + 1) ? LIST_CONSUMERS : 1;
      fa_mbar_init(bar_addr(sb, i), count);
    }
    fa_mbar_init_fence();
    misc[1] = 0;
    misc[2] = 0;
    misc[3] = 0;
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
  // a copy the compiler can see is the same in every lane (read through a broadcast)
  const fa_u32 tmem_u = __shfl_sync(0xffffffffu, tmem, 0);

  if (warp >= 12) fa_setmaxnreg_dec<REGS_OTHER>();

  // Barrier phases: the pair-indexed barriers count the pairs of the CTA across its items (gn);
  // BAR_K, BAR_V, BAR_KFREE, BAR_VFREE, BAR_FINAL and BAR_DKVFREE count the items that have pairs (kvc) - an item
  // without pairs loads no K / V and only has zeros written; the list barriers count all items (itc).
  if (warp == WARP_PRODUCER) {
    // ================================ producer ================================================
    // The whole warp builds the lists; lane 0 issues the loads.
    bool ok = true;
    int gn = 0, kvc = 0;
    int idx = cta;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      // the consumers of the list that was in this buffer two items ago must be done with it
      if (itc >= 2) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFREE + lb), (fa_u32)(((itc >> 1) - 1) & 1), abort_flag);
      if (!ok) break;
      int* pl = pairs + lb * MAXPL;
      const Item it = item_of(min(idx, n_items - 1), p.Hkv, p.B, n_kvt, P.chunk_heads);
      const int hk = it.hk, b = it.b, kt = it.kt;
      int np = -1;
      if (idx < n_items) np = build_pair_list<MAXPL, MAXC>(p, hk, b, kt, G, n_qtiles, (unsigned*)(sm + OFF_CLS), pl, lane);
      if (lane == 0) {
        item[4 * lb] = hk;
        item[4 * lb + 1] = b;
        item[4 * lb + 2] = kt;
        item[4 * lb + 3] = np;
      }
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFULL + lb));
      if (np < 0) break;
      int next = 0;
      if (lane == 0) {
        // the next item is asked for now: the answer is not needed before this item's loads are out
        next = Gd + atomicAdd(P.work_counter, 1);
        const int n0 = kt * BT;
        auto load_tile = [&](const FaTensorMap* map, int off, fa_u32 full, int row, int head) {
          for (int a = 0; a < 2; ++a) fa_tma_load_4d(sb + off + a * ATOM_BYTES, map, full, a * 64, row, head, b);
        };
        for (int n = 0; n < np && ok; ++n, ++gn) {
          const int s = gn % NQS;
          const int pr = pl[n];
          const int m0 = (pr & 0xffff) * BQ, h = hk * G + (pr >> 20);
          // Q tile with the per-row scalars of both halves (prepared by fa_bwd_prep_kernel); one transaction count covers
          // all the copies
          if (gn >= NQS) ok = fa_mbar_wait(bar_addr(sb, BAR_QEMPTY + s), (fa_u32)((gn / NQS - 1) & 1), abort_flag);
          if (!ok) break;
          const long long rbase = ((long long)b * p.Hq + h) * sq_pad + m0;
          const fa_u32 full = bar_addr(sb, BAR_QFULL + s);
          fa_mbar_expect_tx(full, TILE_BYTES + 2 * BQ * 4);
          load_tile(&P.tq, OFF_Q + s * TILE_BYTES, full, m0, h);
          fa_bulk_load(sb + OFF_ROW + s * 2 * BQ * 4, P.nlse2 + rbase, BQ * 4, full);
          fa_bulk_load(sb + OFF_ROW + s * 2 * BQ * 4 + BQ * 4, P.ndelta + rbase, BQ * 4, full);
          if (n == 0) {  // in the order in which the item before lets go of its buffers: V, dO, K
            if (kvc > 0) ok = fa_mbar_wait(bar_addr(sb, BAR_VFREE), (fa_u32)((kvc - 1) & 1), abort_flag);
            if (!ok) break;
            fa_mbar_expect_tx(bar_addr(sb, BAR_V), TILE_BYTES);
            load_tile(&P.tv, OFF_V, bar_addr(sb, BAR_V), n0, hk);
          }
          if (gn > 0) ok = fa_mbar_wait(bar_addr(sb, BAR_DOEMPTY), (fa_u32)((gn - 1) & 1), abort_flag);
          if (!ok) break;
          fa_mbar_expect_tx(bar_addr(sb, BAR_DOFULL), TILE_BYTES);
          load_tile(&P.tdo, OFF_DO, bar_addr(sb, BAR_DOFULL), m0, h);
          if (n == 0) {
            if (kvc > 0) ok = fa_mbar_wait(bar_addr(sb, BAR_KFREE), (fa_u32)((kvc - 1) & 1), abort_flag);
            if (!ok) break;
            fa_mbar_expect_tx(bar_addr(sb, BAR_K), TILE_BYTES);
            load_tile(&P.tk, OFF_K, bar_addr(sb, BAR_K), n0, hk);
          }
        }
        // K and V of the next item are asked into L2 now; their loads can only start when this
        // item is complete, and then they find the tiles close by
        if (ok && next < n_items) {
          const Item i2 = item_of(next, p.Hkv, p.B, n_kvt, P.chunk_heads);
          for (int a = 0; a < 2; ++a) {
            tma_prefetch_l2_4d(&P.tk, a * 64, i2.kt * BT, i2.hk, i2.b);
            tma_prefetch_l2_4d(&P.tv, a * 64, i2.kt * BT, i2.hk, i2.b);
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
    // The whole warp runs the loop and one elected lane issues: with uniform control flow the descriptors live in
    // uniform registers, which makes each tcgen05.mma cheaper to issue than from a single-lane branch.
    const bool leader = fa_elect_one();
    constexpr fa_u32 IDESC_KK = fa_idesc(DT, 128, BQ, 0, 0);  // A, B K-major
    constexpr fa_u32 IDESC_TN = fa_idesc(DT, 128, D, 0, 1);   // A K-major (TMEM), B MN-major
    constexpr fa_u32 IDESC_NN = fa_idesc(DT, 128, D, 1, 1);   // A, B MN-major
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    const fa_u32 loK_k = fa_desc_lo(sb + OFF_K, 16), loV_k = fa_desc_lo(sb + OFF_V, 16);
    const fa_u32 loK_mn = fa_desc_lo(sb + OFF_K, ATOM_BYTES);
    const fa_u32 loDO_k = fa_desc_lo(sb + OFF_DO, 16), loDO_mn = fa_desc_lo(sb + OFF_DO, ATOM_BYTES);
    const fa_u32 loDS_mn = fa_desc_lo(sb + OFF_DS, ATOM_BYTES);
    bool ok = true;
    int gn = 0, kvc = 0;  // gn: the pair whose dS^T comes next
    // S^T = K Q^T (the P^T under it was read by dV of the pair before, issued earlier)
    auto issue_s = [&](int g) {
      const int s = g % NQS;
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_QFULL + s), (fa_u32)((g / NQS) & 1), abort_flag);
      if (!ok) return;
      fa_tc_fence_after();
      const fa_u32 loQ = fa_desc_lo(sb + OFF_Q + s * TILE_BYTES, 16);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        if (leader)
          fa_mma_ss(tmem_u + COL_S, fa_desc_make(loK_k + kstep_kmajor(kk, ATOM_BYTES), HI),
                    fa_desc_make(loQ + kstep_kmajor(kk, ATOM_BYTES), HI), IDESC_KK, kk > 0);
      if (leader) fa_mma_commit(bar_addr(sb, BAR_SFULL));
    };
    // dP^T = V dO^T, over dQ of the pair before, which must have been read; then dV += P^T dO
    auto issue_dp_dv = [&](int g, bool first, bool last) {
      if (g > 0) ok = fa_mbar_wait_all(bar_addr(sb, BAR_DQFREE), (fa_u32)((g - 1) & 1), abort_flag);
      if (ok) ok = fa_mbar_wait_all(bar_addr(sb, BAR_DOFULL), (fa_u32)(g & 1), abort_flag);
      if (!ok) return;
      fa_tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        if (leader)
          fa_mma_ss(tmem_u + COL_DP, fa_desc_make(loV_k + kstep_kmajor(kk, ATOM_BYTES), HI),
                    fa_desc_make(loDO_k + kstep_kmajor(kk, ATOM_BYTES), HI), IDESC_KK, kk > 0);
      if (leader) {
        fa_mma_commit(bar_addr(sb, BAR_DPFULL));
        if (last) fa_mma_commit(bar_addr(sb, BAR_VFREE));
      }
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_PREADY), (fa_u32)(g & 1), abort_flag);
      // the first product of an item overwrites dV (and soon dK): the drain warps must have read the previous item's
      if (ok && first && kvc > 0) ok = fa_mbar_wait_all(bar_addr(sb, BAR_DKVFREE), (fa_u32)((kvc - 1) & 1), abort_flag);
      if (!ok) return;
      fa_tc_fence_after();
      // k-step kk: 16 q columns of P^T, 8 words, the two halves 64 columns apart (each where its threads' scores were)
#pragma unroll
      for (int kk = 0; kk < BQ / 16; ++kk)
        if (leader)
          fa_mma_ts(tmem_u + COL_DV, tmem_u + COL_S + (kk >> 2) * 64 + (kk & 3) * 8, fa_desc_make(loDO_mn + kk * 128, HI), IDESC_TN,
                    (fa_u32)!first | (kk > 0));
      if (leader) fa_mma_commit(bar_addr(sb, BAR_DOEMPTY));
    };
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int np = __shfl_sync(0xffffffffu, item[4 * lb + 3], 0);
      if (leader) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));  // (the issuer needs the count only)
      if (np < 0) break;
      if (np == 0) continue;
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_K), (fa_u32)(kvc & 1), abort_flag);
      if (ok) issue_s(gn);
      if (ok) ok = fa_mbar_wait_all(bar_addr(sb, BAR_V), (fa_u32)(kvc & 1), abort_flag);
      if (ok) issue_dp_dv(gn, true, np == 1);
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const bool more = n + 1 < np;
        if (more) issue_s(gn + 1);
        if (ok) ok = fa_mbar_wait_all(bar_addr(sb, BAR_DSREADY), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        // dK += dS^T Q  (A = dS^T from TMEM, over the dP^T it was computed from)
        const int s = gn % NQS;
        const fa_u32 loQ_mn = fa_desc_lo(sb + OFF_Q + s * TILE_BYTES, ATOM_BYTES);
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk)
          if (leader)
            fa_mma_ts(tmem_u + COL_DK, tmem_u + COL_DP + (kk >> 2) * 64 + (kk & 3) * 8, fa_desc_make(loQ_mn + kk * 128, HI), IDESC_TN,
                      (fa_u32)(n > 0) | (kk > 0));
        if (leader) fa_mma_commit(bar_addr(sb, BAR_QEMPTY + s));
        // dQ = dS K  (A = dS^T read MN-major: M = 128 q, two 64-column atoms; a k-step is 16 kv rows = 2048 bytes of either
        // operand), over dS^T, which dK has read
#pragma unroll
        for (int kk = 0; kk < BT / 16; ++kk)
          if (leader) fa_mma_ss(tmem_u + COL_DP, fa_desc_make(loDS_mn + kk * 128, HI), fa_desc_make(loK_mn + kk * 128, HI), IDESC_NN, kk > 0);
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_DQFULL));
          if (!more) {
            fa_mma_commit(bar_addr(sb, BAR_KFREE));
            fa_mma_commit(bar_addr(sb, BAR_FINAL));
          }
        }
        if (more) issue_dp_dv(gn + 1, false, n + 2 == np);
      }
      ++kvc;
    }
  } else if (warp < 8) {
    // ================================ compute warps ============================================
    fa_setmaxnreg_inc<REGS_COMPUTE>();
    const int half = warp >> 2;               // q columns CW*half .. +CW-1 of the pair tile
    const int lane_base = (warp & 3) * 32;
    const int r = lane_base + lane;           // kv row of this thread inside the tile
    const int c0 = half * CW;                 // first q column of this thread inside the tile
    const fa_u32 tS = tmem + ((fa_u32)lane_base << 16) + COL_S + c0, tD = tmem + ((fa_u32)lane_base << 16) + COL_DP + c0;
    unsigned char* const dsrow = sm + OFF_DS + half * ATOM_BYTES + r * 128;  // (64 columns: one atom per half)
    const float sc2 = p.scale * FA_LOG2E;
    bool ok = true;
    int gn = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int np = item[4 * lb + 3];
      if (np < 0) break;
      const int* pl = pairs + lb * MAXPL;
      const int hk = item[4 * lb], b = item[4 * lb + 1], n0 = item[4 * lb + 2] * BT;
      const int gb = b + p.b_off;
      const int kv = n0 + r;
      const bool row_ok = kv < p.Skv;
      const unsigned* bits = bits_row(p, kv);
      fa_u32 keep[2];  // the mask of this thread's 64 columns, of the next pair from the moment on that this one's is applied
      auto ask = [&](int n) {
        const int pr = pl[n];  // (of pair np: a word behind the list's last, not looked at)
        ask_keep(keep, bits, p, b, hk * G + (pr >> 20), (pr & 0xffff) * BQ + c0, n < np && row_ok && ((pr >> 16) & 0xf) == 1);
      };
      if (FA_HAS_MASK_MOD) ask(0);
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int s = gn % NQS;
        const int pr = pl[n];
        const int m0 = (pr & 0xffff) * BQ, gh = hk * G + (pr >> 20) + p.h_off;
        bool masked = FA_HAS_MASK_MOD && ((pr >> 16) & 0xf) == 1;
        if (!FA_HAS_MASK_MOD) keep[0] = keep[1] = 0xffffffffu;
        if (masked && row_ok && bits == nullptr) eval_keep(keep, gb, gh, m0 + c0, kv);
        masked |= clear_beyond(keep, p.Sq - (m0 + c0));
        const fa_u32 live = live_steps(keep, masked, row_ok);
        const float* rowp = (const float*)(sm + OFF_ROW + s * 2 * BQ * 4) + c0;
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_QFULL + s), (fa_u32)((gn / NQS) & 1), abort_flag);
        if (ok) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_SFULL), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        // The columns come in steps of 16, the load of a step in flight while the previous one is computed.  P^T of a step
        // takes 8 of the 16 columns its own or an earlier step's scores were read from.
        float pg[CW];
        {
          float sA[16], sB[16];
          fa_u32 p8[8];
          fa_tmem_ld16(tS, sA);
          fa_tmem_wait_ld();
#define FA_STEP(CUR, NEXT, C)                                                                                      \
  if ((C) + 16 < CW) fa_tmem_ld16(tS + (C) + 16, NEXT);                                                            \
  if (FA_BWD_MASKS ? (live >> ((C) / 16)) & 1u : row_ok) {                                                  \
    p_chunk(CUR, rowp + (C), p8, pg + (C), masked, keep[(C) >> 5] >> ((C) & 31), m0 + c0 + (C), kv, gb, gh, p.scale, sc2); \
  } else {                                                                                                         \
    _Pragma("unroll") for (int e = 0; e < 8; ++e) p8[e] = 0u;                                                      \
    _Pragma("unroll") for (int e = 0; e < 16; ++e) pg[(C) + e] = 0.f;                                              \
  }                                                                                                                \
  if ((C) + 16 < CW) fa_tmem_wait_ld();                                                                            \
  fa_tmem_st8(tS + (C) / 2, p8);
          FA_STEP(sA, sB, 0)
          FA_STEP(sB, sA, 16)
          FA_STEP(sA, sB, 32)
          FA_STEP(sB, sA, 48)
#undef FA_STEP
        }
        fa_tmem_wait_st();
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_PREADY));
        if (FA_HAS_MASK_MOD) ask(n + 1);
        // dP^T is there: and dS^T of the pair before is not read any more (the order of issue)
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DPFULL), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        {
          float dA[16], dB[16];
          fa_u32 d8[8];
          fa_tmem_ld16(tD, dA);
          fa_tmem_wait_ld();
          // dS^T row r, to TMEM in the way of P^T and to shared memory: 16-byte chunk k of a 128-byte atom row goes to
          // position k ^ (r & 7) (the 128-byte swizzle of the operand layout)
#define FA_STEP(CUR, NEXT, C)                                                                                      \
  if ((C) + 16 < CW) fa_tmem_ld16(tD + (C) + 16, NEXT);                                                            \
  if (FA_BWD_MASKS ? (live >> ((C) / 16)) & 1u : row_ok) {                                                  \
    ds_chunk(CUR, rowp + BQ + (C), pg + (C), d8);                                                                  \
  } else {                                                                                                         \
    _Pragma("unroll") for (int e = 0; e < 8; ++e) d8[e] = 0u;                                                      \
  }                                                                                                                \
  *(uint4*)(dsrow + ((((C) / 8) ^ (r & 7)) * 16)) = make_uint4(d8[0], d8[1], d8[2], d8[3]);                        \
  *(uint4*)(dsrow + ((((C) / 8 + 1) ^ (r & 7)) * 16)) = make_uint4(d8[4], d8[5], d8[6], d8[7]);                    \
  if ((C) + 16 < CW) fa_tmem_wait_ld();                                                                            \
  fa_tmem_st8(tD + (C) / 2, d8);
          FA_STEP(dA, dB, 0)
          FA_STEP(dB, dA, 16)
          FA_STEP(dA, dB, 32)
          FA_STEP(dB, dA, 48)
#undef FA_STEP
        }
        fa_tmem_wait_st();
        fence_proxy_async();
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_DSREADY));
      }
      if (!ok) break;
      // every lane has read its last list entry: the list may be overwritten
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
    }
  } else if (warp < 12) {
    // ================================ drain warps: dQ of every pair, dK / dV of every item =======
    fa_setmaxnreg_inc<REGS_DRAIN>();
    const int lane_base = (warp & 3) * 32;
    const int r = lane_base + lane;  // TMEM lane: q row of the pair; kv row for dK / dV
    const fa_u32 t_lane = tmem + ((fa_u32)lane_base << 16);
    const int dtid = tid - 256;
    unsigned char* const strow = sm + OFF_ST + r * 128;  // this thread's row of the staging buffer
    bool ok = true;
    int gn = 0, kvc = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      // The four drain warps meet at named barriers, so they have to leave their loops together: a
      // warp whose wait failed says so in a flag only the drain warps write, joins the next named
      // barrier like the others, and all four read the flag behind that barrier.
      ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) misc[3] = 1;
      named_bar_sync(1, 128);
      if (misc[3] != 0) {
        ok = false;
        break;
      }
      const int np = item[4 * lb + 3];
      if (np < 0) break;  // (the same in all four warps)
      const int* pl = pairs + lb * MAXPL;
      const int hk = item[4 * lb], b = item[4 * lb + 1], n0 = item[4 * lb + 2] * BT;
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int pr = pl[n];
        const int qt = pr & 0xffff, h = hk * G + (pr >> 20);
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DQFULL), (fa_u32)(gn & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        // The whole row comes into registers, so that the columns are free at once; it leaves by 32 columns through the
        // warp's own 4 KB of staging, each time one bulk reduce-add of 4 KB (no barrier between the warps).  16-byte chunk k of
        // lane r goes to position k ^ (r & 7), which spreads the rows over the banks.  (red.global.add.v4 straight from the
        // registers, 512 consecutive bytes per warp: dense B4 H8 S4096 676 us against 582.)
        float* gdst = P.dq_acc + (((long long)b * p.Hq + h) * n_qtiles + qt) * (128 * D) + (warp & 3) * 1024;
        float a[D / 32][32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) fa_tmem_ld32(t_lane + COL_DP + 32 * c, a[c]);
        fa_tmem_wait_ld();
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_DQFREE));
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          if (lane == 0) bulk_wait_read0();  // the previous reduce (or store) has read the staging buffer
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            *(float4*)(strow + ((k ^ (r & 7)) * 16)) = make_float4(a[c][4 * k], a[c][4 * k + 1], a[c][4 * k + 2], a[c][4 * k + 3]);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            bulk_reduce_add_f32(gdst + c * 4096, sb + OFF_ST + (warp & 3) * 4096, 4096);
            bulk_commit();
          }
        }
      }
      // ---- dK (scaled) and dV of the item.  A thread owns one kv row (TMEM lane); 64 columns at a
      // time are converted into the staging buffer in the layout of a K tile (128-byte rows, 16-byte
      // chunk k of row r at k ^ (r & 7)) and leave through one tensor-map store, which writes whole
      // lines and clips the rows beyond Skv.  An item without pairs has zeros written.
      if (np > 0) {
        if (ok) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_FINAL), (fa_u32)(kvc & 1), abort_flag);
        if (!ok) misc[3] = 1;
        named_bar_sync(1, 128);
        if (misc[3] != 0) {
          ok = false;
          break;
        }
        fa_tc_fence_after();
#pragma unroll 1
        for (int part = 0; part < 4; ++part) {
          const int which = part >> 1, a = part & 1;  // dK atoms first, then dV
          const float mul = which == 0 ? p.scale : 1.f;
          // the previous reduces and stores must have finished reading the staging buffer
          if (lane == 0) bulk_wait_read0();
          named_bar_sync(1, 128);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            float o[32];
            fa_tmem_ld32(t_lane + (which == 0 ? COL_DK : COL_DV) + a * 64 + c * 32, o);
            fa_tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
              uint4 w;
              w.x = fa_pack2<DT>(o[e] * mul, o[e + 1] * mul);
              w.y = fa_pack2<DT>(o[e + 2] * mul, o[e + 3] * mul);
              w.z = fa_pack2<DT>(o[e + 4] * mul, o[e + 5] * mul);
              w.w = fa_pack2<DT>(o[e + 6] * mul, o[e + 7] * mul);
              *(uint4*)(strow + (((4 * c + (e >> 3)) ^ (r & 7)) * 16)) = w;
            }
          }
          if (part == 3) {
            // dK and dV are out of TMEM: the next item's first products may overwrite them
            fa_tc_fence_before();
            fa_mbar_arrive(bar_addr(sb, BAR_DKVFREE));
          }
          fence_proxy_async();
          named_bar_sync(1, 128);
          if (dtid == 0) {
            fa_tma_store_4d(which == 0 ? &P.tdk : &P.tdv, sb + OFF_ST, a * 64, n0, hk, b);
            bulk_commit();
          }
        }
        // (the staging buffer is the warps' own again once the last store has read it)
        if (dtid == 0) bulk_wait_read0();
        named_bar_sync(1, 128);
        ++kvc;
      } else {
        // an item without pairs: zeros, straight from the registers (rare; a row per thread)
        const int kv = n0 + r;
        if (kv < p.Skv) {
#pragma unroll
          for (int which = 0; which < 2; ++which) {
            const FaTensor& dst = which == 0 ? p.dk : p.dv;
            char* og = (char*)dst.ptr + ((long long)b * dst.sb + (long long)hk * dst.sh + (long long)kv * dst.ss) * 2;
            for (int c = 0; c < D / 8; ++c) *(uint4*)(og + c * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
      }
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
    }
    if (lane == 0) bulk_wait0();
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
