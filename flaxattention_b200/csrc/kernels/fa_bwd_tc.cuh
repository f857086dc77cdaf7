// Flash-attention backward for sm_100a on the 5th-generation tensor cores (fp16 / bf16,
// D = Dv = 64; D = 128: fa_bwd_tc128.cuh).  One kernel computes dK, dV and dQ in a single pass over the
// (kv tile, q tile) pairs the BlockMask lists: five tcgen05.mma products per pair and one
// exponential per score, where the two-scan reference kernel
// (flaxattention/kernel/attention.py:423-553) and fa_bwd.cuh need seven products and two
// exponentials.
//
// The unit of work (an item) is a 128-row kv tile of one (batch, kv head) together with the q tiles
// of the query heads that share it.  The kernel is persistent: one CTA per SM, every CTA works
// through items it takes from a counter in global memory, and TMEM and the barriers are set up
// once per CTA.  A pair is 128 kv rows x 128 query rows.  Everything is kept transposed so that dK and dV
// have kv rows (TMEM lanes) and P^T can be fed to the tensor core straight from TMEM:
//   1. S^T  = K Q^T                      (TMEM, 128 kv x 128 q, fp32)
//   2. dP^T = V dO^T                     (TMEM)
//      p = 2^(x - lse), ds = p (dp - delta) score_mod'      thread (kv row, 64 q columns)
//      P^T -> TMEM (16 bit),  dS^T -> shared memory (16 bit, [kv][q], 128-byte swizzle)
//   3. dV += P^T dO                      (A from TMEM)
//   4. dK += dS^T Q                      (A = dS^T from smem, K-major)
//   5. dQ = dS K                         (A = the same dS^T tile read MN-major, B = K; 128 q x 64 d)
// The dQ tile of a pair leaves warp by warp, 32 columns at a time, through 4 KB of staging and a bulk reduce-add each, into
// an fp32 accumulation buffer (summation order over kv tiles is not fixed; a small kernel scales, un-permutes and
// converts it afterwards).
// dK and dV are written once per item.
//
// Warp roles (16 warps): 0-3 and 4-7 compute (first / second half of the q columns of the pair),
// 8-11 drain (dQ of every pair, dK / dV of every item), 12 producer (pair lists and TMA loads), 13 MMA issuer A (products 1-2, TMEM owner), 14 MMA issuer B
// (products 3-4), 15 MMA issuer C (product 5).
// S^T/dP^T of pair n+1 are issued as soon as the compute warps hold pair n in registers, so
// the tensor core runs ahead of the element-wise work.
//
// TMEM (512 columns): S^T 0-127, dP^T 128-255, P^T 256-319, dV 320-383, dK 384-447, dQ 448-511
// Every mbarrier wait is bounded (see fa_sm100.cuh).
//
// Compile-time parameters (macros): FA_DTYPE (0 fp16, 1 bf16), FA_BWD_KV2 (two K / V buffers and one of dS^T instead of
// one and two).
#pragma once
#include "fa_bwd_items.cuh"

namespace fa_btc {
using namespace fa_bwd_items;

constexpr int DT = FA_DTYPE;
constexpr int D = 64;
constexpr int BT = 128;                    // kv rows of a tile
constexpr int BQ = 128;                    // q rows of a pair
constexpr int CW = BQ / 2;                 // q columns of one compute thread
constexpr int TILE_BYTES = 128 * 128;      // a K, V, Q or dO tile: 128 rows x 128 bytes (64 values)
// K / V and dS^T buffers.  The pace of a pair is set by the hand-over of P^T and dS^T: with one dS^T buffer the
// compute warps may store pair n + 1 only when products 3-5 of pair n are complete.  With two they wait for
// product 3 of pair n (issued first) and, by the order of issue, products 4-5 of pair n - 1, which is
// long past; the Q / dO ring gives up its fourth stage for it.  Measured against one buffer and four
// stages, backward alone, us: dense B8 H8 S2048 231 -> 225, B4 H16/4 S2048 251 -> 239.
// Shared memory holds, instead of the second dS^T buffer, a second K / V buffer (FA_BWD_KV2): K and V of
// the next item are loaded while the current one is computed and nothing waits at the change of items, which pays
// when items are short or uneven.  The host picks (bwd_tc_kv2).
#ifndef FA_BWD_KV2
#define FA_BWD_KV2 0
#endif
constexpr int KVBUF = FA_BWD_KV2 ? 2 : 1;
constexpr int NSTAGE = 3;
constexpr int NDS = KVBUF == 1 ? 2 : 1;                // dS^T buffers
constexpr int DS_BYTES = 2 * TILE_BYTES;               // dS^T: [128 kv][128 q] as two blocks of 64 q columns
constexpr int MAXPL = 1024;              // (head, q tile) pairs of one item (two such lists fit in shared memory)
constexpr int MAXC = 256;                // 128-row q tiles per head (Sq <= 32768)
constexpr int NT = 512;
constexpr int WARP_PRODUCER = 12, WARP_MMA = 13, WARP_MMA_B = 14, WARP_MMA_C = 15;
// Register split (setmaxnreg): the kernel starts with 128 registers per thread (65536 / 512).  The drain warps hold a row of dQ
// (64 values, so that its TMEM columns are free after one round of loads) and give up 16 each, producer and issuers 32, and the eight
// compute warps take 24 each; an increase that asked for more than the decrease releases would wait forever.  160 / 96 / 96 is as
// fast (causal B2 H16/4 S3001 224.6 / 226.9 us, attention sink B2 H8 S8192 186 / 187); with 56 for all but the compute warps these
// spilled, and the kernel was 4-5 % slower.  What is left of spills is 8 to 20 bytes of scalars, with either split.
constexpr int REGS_COMPUTE = 152, REGS_DRAIN = 112, REGS_OTHER = 96;
static_assert(2 * REGS_COMPUTE + REGS_DRAIN + REGS_OTHER <= 4 * 128, "setmaxnreg.inc would wait forever");

// shared memory map (from a 1024-byte aligned base)
constexpr int OFF_K = 0;
constexpr int OFF_V = OFF_K + KVBUF * TILE_BYTES;
constexpr int OFF_Q = OFF_V + KVBUF * TILE_BYTES;             // NSTAGE tiles
constexpr int OFF_DO = OFF_Q + NSTAGE * TILE_BYTES;            // NSTAGE tiles
constexpr int OFF_DS = OFF_DO + NSTAGE * TILE_BYTES;           // dS^T
constexpr int OFF_DQ = OFF_DS + NDS * DS_BYTES;      // fp32 staging 128 x 32, 4 KB of each drain warp
constexpr int DQ_HALF_BYTES = 128 * 32 * 4;
constexpr int OFF_ROW = OFF_DQ + DQ_HALF_BYTES;             // NSTAGE x (nlse2[BQ], ndelta[BQ]) floats
constexpr int OFF_BAR = OFF_ROW + NSTAGE * 2 * BQ * 4;
constexpr int NBARS = 2 + 3 * NSTAGE + 15;
constexpr int OFF_MISC = OFF_BAR + NBARS * 8;               // tmem base, abort, -, drain flag
constexpr int OFF_ITEM = OFF_MISC + 16;                     // int item[2][4]: kv head (KV2: item number), batch, kv tile, pairs (-1: no more work)
constexpr int OFF_PAIR = OFF_ITEM + 32;                     // int pair[2][MAXPL]: q tile | mode << 16 | g << 20
constexpr int OFF_CLS = OFF_PAIR + 2 * MAXPL * 4;           // unsigned cls[2][MAXC / 32] (scratch of the list builder)
constexpr int SMEM_BYTES = OFF_CLS + 2 * MAXC / 8 + 1024;
// (the pointers of up to eight captured buffers are static shared memory beside this)
static_assert(SMEM_BYTES + 8 * 8 <= 227 * 1024, "shared memory");
constexpr int TMEM_COLS = 512;
constexpr int COL_S = 0, COL_DP = BQ, COL_P = 2 * BQ;
constexpr int COL_DV = 320, COL_DK = 384, COL_DQ = 448;

constexpr int BAR_KV = 0;                   // [2] K and V of an item have landed in buffer kb
// A stage's Q tile (with the row scalars) and dO tile are released separately: dO is last read by
// product 3, Q by product 4, and the sooner a slot is free the further ahead the producer runs.
constexpr int BAR_QFULL = 2, BAR_QEMPTY = 2 + NSTAGE, BAR_DOEMPTY = 2 + 2 * NSTAGE;
constexpr int BAR_SFULL = 2 + 3 * NSTAGE;   // S^T and dP^T of a pair are in TMEM
constexpr int BAR_SFREE = BAR_SFULL + 1;    // compute warps hold them in registers (256 arrivals)
constexpr int BAR_PREADY = BAR_SFULL + 2;   // P^T in TMEM and dS^T in smem (256 arrivals)
constexpr int BAR_PFREE = BAR_SFULL + 3;    // P^T and the next dS^T buffer may be written (see NDS)
constexpr int BAR_DQFULL = BAR_SFULL + 4;   // dQ of the pair is in TMEM
constexpr int BAR_DQFREE = BAR_SFULL + 5;   // drain warps hold it in registers (128 arrivals)
constexpr int BAR_FINAL = BAR_SFULL + 6;    // [2] products 3-5 of the last pair of the item in buffer kb are complete
constexpr int BAR_DKVFREE = BAR_SFULL + 8;  // the drain warps have read dK and dV of an item out of TMEM (128 arrivals)
constexpr int BAR_LISTFULL = BAR_SFULL + 9; // [2] the producer has published an item and its pair list
constexpr int BAR_LISTFREE = BAR_SFULL + 11;  // [2] the 15 consumers of a list are done with it
constexpr int BAR_KVFREE = BAR_SFULL + 13;  // [2] (two K / V buffers) the stores of dK / dV staged in buffer kb have read it
constexpr int LIST_CONSUMERS = 3 + 8 + 4;   // MMA issuers, compute warps, drain warps (one arrival each)

__device__ __forceinline__ fa_u32 bar_addr(fa_u32 sb, int i) { return sb + OFF_BAR + i * 8; }

// Element-wise work of one thread on a W-column chunk: scores s and dp (fp32, raw) for kv row
// `kv` and q columns q0 .. q0+W-1 -> packed P^T and dS^T (16 bit).  q0 is a multiple of W (the
// compiler can see that from how the caller builds it), so the low bits of every q index are
// compile-time constants inside the mods while one copy of this code serves all chunks of a
// tile row.  nlse2 / ndelta point at the row scalars of column q0.
template <int W>
__device__ __forceinline__ void chunk(const float (&s)[W], const float (&dp)[W], const float* nlse2, const float* ndelta,
                                      fa_u32 (&pp)[W / 2], fa_u32 (&ds)[W / 2], int q0, int kv, int gb, int gh,
                                      float scale, float sc2) {
#if !FA_HAS_SCORE_MOD || defined(FA_SCORE_AFFINE)
  // no score_mod, or an affine one: two elements per instruction (packed fp32) wherever the
  // hardware has the form; only the exponentials are per element, and the rounding of the raw scores where it is asked for
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_LINEAR_Q)
  // the multiplier does not read q and the bias is linear in it (relative-position biases such as
  // ALiBi): both are taken once, at the first column of the chunk; every eighth column is reached from there with one FMA,
  // the ones behind it by adding multiples of the slope that are kept (column numbers as packed constants would take two
  // moves per pair; without a mask, a kernel with registers to spare, they are the faster form: B2 H2/1 S3044 forward and
  // backward 126.6 against 128.3 us, causal B8 H8 S2048 228 with this form against 233).  A derivative of 1 is not multiplied with.
  const float lin_g = fa_score_mul(0.f, gb, gh, q0, kv);
  const fa_u64 lin_g2 = fa_f2(lin_g, lin_g), lin_gs2 = fa_f2(lin_g * sc2, lin_g * sc2);
  const float lin_base = fa_score_add2(0.f, gb, gh, q0, kv), lin_dq = fa_score_add2_dq(0.f, gb, gh, q0, kv);
#if !FA_HAS_MASK_MOD
  const fa_u64 lin_b2 = fa_f2(lin_base, lin_base), lin_d2 = fa_f2(lin_dq, lin_dq);
#endif
  [[maybe_unused]] const fa_u64 lin_od[4] = {fa_f2(0.f, lin_dq), fa_f2(2.f * lin_dq, 3.f * lin_dq), fa_f2(4.f * lin_dq, 5.f * lin_dq), fa_f2(6.f * lin_dq, 7.f * lin_dq)};
  [[maybe_unused]] float at8 = lin_base;
#endif
#pragma unroll
  for (int e = 0; e < W; e += 4) {
    const float4 nl = *(const float4*)(nlse2 + e);
    const float4 nd = *(const float4*)(ndelta + e);
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      const int qi0 = q0 | (e + u), qi1 = q0 | (e + u + 1);
      const fa_u64 nl2 = u == 0 ? fa_f2(nl.x, nl.y) : fa_f2(nl.z, nl.w);
      const fa_u64 nd2 = u == 0 ? fa_f2(nd.x, nd.y) : fa_f2(nd.z, nd.w);
      float s0 = s[e + u], s1 = s[e + u + 1];
#if FA_ROUND_SCORES
      fa_round2<DT>(s0, s1);
#endif
      const fa_u64 s2 = fa_f2(s0, s1);
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_LINEAR_Q)
      [[maybe_unused]] const fa_u64 g2 = lin_g2;
#if !FA_HAS_MASK_MOD
      const fa_u64 b2 = fa_add2(fa_fma2(fa_f2((float)(e + u), (float)(e + u + 1)), lin_d2, lin_b2), nl2);
#else
      if (e > 0 && (e + u) % 8 == 0) at8 = fmaf((float)(e + u), lin_dq, lin_base);
      const fa_u64 b2 = fa_add2(fa_add2(fa_f2(at8, at8), nl2), lin_od[((e + u) % 8) / 2]);  // (large ones first: they cancel)
#endif
      const fa_u64 x2 = fa_fma2(s2, lin_gs2, b2);
#elif FA_HAS_SCORE_MOD
      const fa_u64 g2 = fa_f2(fa_score_mul(0.f, gb, gh, qi0, kv), fa_score_mul(0.f, gb, gh, qi1, kv));
      const fa_u64 b2 = fa_add2(fa_f2(fa_score_add2(0.f, gb, gh, qi0, kv), fa_score_add2(0.f, gb, gh, qi1, kv)), nl2);
      const fa_u64 x2 = fa_fma2(s2, fa_mul2(g2, fa_f2(sc2, sc2)), b2);
#else
      const fa_u64 x2 = fa_fma2(s2, fa_f2(sc2, sc2), nl2);
#endif
      float x0, x1;
      fa_f2_unpack(x2, x0, x1);
      const float p0 = fa_ex2(x0), p1 = fa_ex2(x1);
      fa_u64 d2 = fa_mul2(fa_f2(p0, p1), fa_add2(fa_f2(dp[e + u], dp[e + u + 1]), nd2));
#if FA_HAS_SCORE_MOD && !defined(FA_SCORE_MUL_ONE)
      d2 = fa_mul2(d2, g2);
#endif
      float d0, d1;
      fa_f2_unpack(d2, d0, d1);
      pp[(e + u) / 2] = fa_pack2<DT>(p0, p1);
      ds[(e + u) / 2] = fa_pack2<DT>(d0, d1);
    }
  }
#else
#pragma unroll
  for (int e = 0; e < W; e += 4) {
    const float4 nl = *(const float4*)(nlse2 + e);
    const float4 nd = *(const float4*)(ndelta + e);
    float pv[4], dv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int qi = q0 | (e + u);
      const float nlu = u == 0 ? nl.x : (u == 1 ? nl.y : (u == 2 ? nl.z : nl.w));
      const float ndu = u == 0 ? nd.x : (u == 1 ? nd.y : (u == 2 ? nd.z : nd.w));
      float x = s[e + u];
#if FA_ROUND_SCORES
      {
        float dummy = 0.f;
        fa_round2<DT>(x, dummy);
      }
#endif
      const float g = fa_score_mod_grad(x * scale, gb, gh, qi, kv);
      x = fa_score_mod(x * scale, gb, gh, qi, kv) * FA_LOG2E + nlu;
      const float pr = fa_ex2(x);
      pv[u] = pr;
      dv[u] = pr * (dp[e + u] + ndu) * g;
    }
    pp[e / 2] = fa_pack2<DT>(pv[0], pv[1]);
    pp[e / 2 + 1] = fa_pack2<DT>(pv[2], pv[3]);
    ds[e / 2] = fa_pack2<DT>(dv[0], dv[1]);
    ds[e / 2 + 1] = fa_pack2<DT>(dv[2], dv[3]);
  }
#endif
}


// Item number -> (kv head, batch, kv tile): with one K / V buffer by chunks of heads (fa_bwd_items::item_of), with two heads
// fastest and the kv tile slowest (there the items are short and the time to their first loads counts, causal
// B1 H8 S8192 228 -> 242 us).
__device__ __forceinline__ Item item_at(int idx, int Hkv, int B, int n_kvt, int ch) {
  if (KVBUF == 2) return {idx % Hkv, (idx / Hkv) % B, idx / (Hkv * B)};
  return item_of(idx, Hkv, B, n_kvt, ch);
}

// What the producer has published of an item.  With two K / V buffers that is the item's number, `idx`, which the
// callers read together with the number of pairs and which is taken apart here: reading the three parts made the
// compute warps spill and the kernel 4 % slower (causal B1 H8 S8192 D64 230 -> 241 us).
__device__ __forceinline__ Item read_item(int idx, const volatile int* item, int Hkv, int B) {
  if (KVBUF == 2) return {idx % Hkv, (idx / Hkv) % B, idx / (Hkv * B)};
  return {item[0], item[1], item[2]};
}

}  // namespace fa_btc

extern "C" __global__ void __launch_bounds__(fa_btc::NT, 1) fa_bwd_tc_kernel(const __grid_constant__ FaBwdTcParams P) {
  using namespace fa_btc;
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
  const int n_ctiles = min((p.Sq + 127) / 128, MAXC);  // 128-row q tiles (the grain of the BlockMask walk)
  const int sq_pad = ((p.Sq + 127) / 128) * 128;
  const int n_kvt = (p.Skv + BT - 1) / BT;
  const int n_items = p.Hkv * p.B * n_kvt;
  const int Gd = (int)gridDim.x, cta = (int)blockIdx.x;

  volatile int* misc = (volatile int*)(sm + OFF_MISC);  // [0] tmem base, [1] abort, [2] unused, [3] drain warps leave
  int* pairs = (int*)(sm + OFF_PAIR);                   // two lists of MAXPL pairs
  volatile int* item = (volatile int*)(sm + OFF_ITEM);  // per list: kv head, batch, kv tile, pairs

  // An item is the 128-row kv tile of one (batch, kv head); items are numbered so that the
  // heaviest come early and heads stay together (item_of).  The kernel is
  // persistent: CTA c starts with item c and takes further items from a counter in global memory,
  // so TMEM, the barriers and the descriptors are set up once per CTA, the loads of an item run
  // under the tail of the one before, and the CTAs stay level whatever the mask does to the work
  // per item.  The producer warp builds the pair list of the next item (two lists in shared
  // memory) while the others work on the current one.

  // ---- set-up --------------------------------------------------------------------------------
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      fa_mbar_init(bar_addr(sb, BAR_KV + i), 1);
      fa_mbar_init(bar_addr(sb, BAR_FINAL + i), 2);  // products 3-4 and product 5 of an item's last pair
      fa_mbar_init(bar_addr(sb, BAR_KVFREE + i), 1);
    }
    for (int s = 0; s < NSTAGE; ++s) {
      fa_mbar_init(bar_addr(sb, BAR_QFULL + s), 1);
      fa_mbar_init(bar_addr(sb, BAR_QEMPTY + s), 2);  // one arrival from each MMA issuer
      fa_mbar_init(bar_addr(sb, BAR_DOEMPTY + s), 2);
    }
    fa_mbar_init(bar_addr(sb, BAR_SFULL), 1);
    fa_mbar_init(bar_addr(sb, BAR_SFREE), 256);
    fa_mbar_init(bar_addr(sb, BAR_PREADY), 256);
    fa_mbar_init(bar_addr(sb, BAR_PFREE), 2);  // one arrival from each of the issuers of products 3-4 and 5
    fa_mbar_init(bar_addr(sb, BAR_DQFULL), 1);
    fa_mbar_init(bar_addr(sb, BAR_DQFREE), 128);
    fa_mbar_init(bar_addr(sb, BAR_DKVFREE), 128);
    for (int i = 0; i < 2; ++i) {
      fa_mbar_init(bar_addr(sb, BAR_LISTFULL + i), 1);
      fa_mbar_init(bar_addr(sb, BAR_LISTFREE + i), LIST_CONSUMERS);
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
  else if (warp >= 8) fa_setmaxnreg_dec<REGS_DRAIN>();

  // Barrier phases: the pair-indexed barriers count the pairs of the CTA across its items (gn);
  // BAR_KV, BAR_FINAL and BAR_DKVFREE count the items that have pairs (kvc) - an item without
  // pairs loads no K / V and only has zeros written; the list barriers count all items (itc).
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
      const Item it = item_at(min(idx, n_items - 1), p.Hkv, p.B, n_kvt, P.chunk_heads);
      const int hk = it.hk, b = it.b, kt = it.kt;
      int np = -1;
      if (idx < n_items) np = build_pair_list<MAXPL, MAXC>(p, hk, b, kt, G, n_ctiles, (unsigned*)(sm + OFF_CLS), pl, lane);
      if (lane == 0) {
        item[4 * lb] = KVBUF == 2 ? idx : hk;
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
        // The K / V buffers are free once the last products of the previous item are complete;
        // the Q / dO slots of the item's first pairs free up earlier, so those loads go first.
        const int kb = kvc % KVBUF, use = kvc / KVBUF;
        const int kvpos = (KVBUF == 2 || kvc == 0) ? 0 : min(NSTAGE, np) - 1;
        for (int n = 0; n < np && ok; ++n, ++gn) {
          if (n == kvpos) {
            if (use > 0) ok = fa_mbar_wait(bar_addr(sb, (KVBUF == 2 ? BAR_KVFREE : BAR_FINAL) + kb), (fa_u32)((use - 1) & 1), abort_flag);
            if (!ok) break;
            const fa_u32 full = bar_addr(sb, BAR_KV + kb);
            fa_mbar_expect_tx(full, 2 * TILE_BYTES);
            fa_tma_load_4d(sb + OFF_K + kb * TILE_BYTES, &P.tk, full, 0, n0, hk, b);
            fa_tma_load_4d(sb + OFF_V + kb * TILE_BYTES, &P.tv, full, 0, n0, hk, b);
          }
          const int s = gn % NSTAGE;
          const fa_u32 ph = (fa_u32)((gn / NSTAGE) & 1);
          const int pr = pl[n];
          const int m0 = (pr & 0xffff) * BQ, h = hk * G + (pr >> 20);
          if (gn >= NSTAGE) ok = fa_mbar_wait(bar_addr(sb, BAR_DOEMPTY + s), ph ^ 1u, abort_flag);
          if (!ok) break;
          // Q and dO tiles plus the per-row scalars of the q tile (prepared by fa_bwd_prep_kernel);
          // one transaction count covers all the copies
          const long long rbase = ((long long)b * p.Hq + h) * sq_pad + m0;
          const fa_u32 full = bar_addr(sb, BAR_QFULL + s);
          fa_mbar_expect_tx(full, 2 * TILE_BYTES + 2 * BQ * 4);
          fa_tma_load_4d(sb + OFF_DO + s * TILE_BYTES, &P.tdo, full, 0, m0, h, b);
          if (gn >= NSTAGE) ok = fa_mbar_wait(bar_addr(sb, BAR_QEMPTY + s), ph ^ 1u, abort_flag);
          if (!ok) break;
          fa_tma_load_4d(sb + OFF_Q + s * TILE_BYTES, &P.tq, full, 0, m0, h, b);
          fa_bulk_load(sb + OFF_ROW + s * 2 * BQ * 4, P.nlse2 + rbase, BQ * 4, full);
          fa_bulk_load(sb + OFF_ROW + s * 2 * BQ * 4 + BQ * 4, P.ndelta + rbase, BQ * 4, full);
        }
        // K and V of the next item are asked into L2 now; their loads can only start when this
        // item is complete, and then they find the tiles close by
        if (KVBUF == 1 && ok && next < n_items) {
          const Item i2 = item_at(next, p.Hkv, p.B, n_kvt, P.chunk_heads);
          const int hk2 = i2.hk, b2 = i2.b, n2 = i2.kt * BT;
          tma_prefetch_l2_4d(&P.tk, 0, n2, hk2, b2);
          tma_prefetch_l2_4d(&P.tv, 0, n2, hk2, b2);
        }
      }
      if (np > 0) ++kvc;
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      gn = __shfl_sync(0xffffffffu, gn, 0);
      idx = __shfl_sync(0xffffffffu, next, 0);
    }
  } else if (warp == WARP_MMA) {
    // ================================ MMA issuer A: products 1-2 ===============================
    // (several issuing warps, so that the waits of one overlap the issue of the other; warp A also
    //  owns the TMEM allocation).  The whole warp runs the loop and one elected lane issues: with
    //  uniform control flow the descriptors live in uniform registers, which makes each
    //  tcgen05.mma cheaper to issue than from a single-lane branch, and the issue rate of this
    //  one thread is what bounds the tensor core here.
    const bool leader = fa_elect_one();
    constexpr fa_u32 IDESC_KK = fa_idesc(DT, 128, BQ, 0, 0);  // A, B K-major, N = BQ
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    bool ok = true;
    int gn = 0, kvc = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int np = __shfl_sync(0xffffffffu, item[4 * lb + 3], 0);
      if (leader) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));  // (the issuers need the count only)
      if (np < 0) break;
      if (np == 0) continue;
      const int kb = kvc % KVBUF;
      const fa_u32 loK_k = fa_desc_lo(sb + OFF_K + kb * TILE_BYTES, 16), loV_k = fa_desc_lo(sb + OFF_V + kb * TILE_BYTES, 16);
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_KV + kb), (fa_u32)((kvc / KVBUF) & 1), abort_flag);
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int s = gn % NSTAGE;
        ok = fa_mbar_wait_all(bar_addr(sb, BAR_QFULL + s), (fa_u32)((gn / NSTAGE) & 1), abort_flag);
        if (ok && gn > 0) ok = fa_mbar_wait_all(bar_addr(sb, BAR_SFREE), (fa_u32)((gn - 1) & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        const fa_u32 loQ = fa_desc_lo(sb + OFF_Q + s * TILE_BYTES, 16), loDO = fa_desc_lo(sb + OFF_DO + s * TILE_BYTES, 16);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          if (leader)
            fa_mma_ss(tmem_u + COL_S, fa_desc_make(loK_k + kstep_kmajor(kk, TILE_BYTES), HI),
                      fa_desc_make(loQ + kstep_kmajor(kk, TILE_BYTES), HI), IDESC_KK, kk > 0);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          if (leader)
            fa_mma_ss(tmem_u + COL_DP, fa_desc_make(loV_k + kstep_kmajor(kk, TILE_BYTES), HI),
                      fa_desc_make(loDO + kstep_kmajor(kk, TILE_BYTES), HI), IDESC_KK, kk > 0);
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_SFULL));
          fa_mma_commit(bar_addr(sb, BAR_QEMPTY + s));  // first of the two arrivals that free each tile of the stage
          fa_mma_commit(bar_addr(sb, BAR_DOEMPTY + s));
        }
      }
      ++kvc;
    }
  } else if (warp == WARP_MMA_B) {
    // ================================ MMA issuer B: products 3-4 ===============================
    const bool leader = fa_elect_one();
    constexpr fa_u32 IDESC_TN = fa_idesc(DT, 128, D, 0, 1);    // A K-major (TMEM or smem), B MN-major, N = D
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    bool ok = true;
    int gn = 0, kvc = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int np = __shfl_sync(0xffffffffu, item[4 * lb + 3], 0);
      if (leader) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
      if (np < 0) break;
      if (np == 0) continue;
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int s = gn % NSTAGE;
        ok = fa_mbar_wait_all(bar_addr(sb, BAR_PREADY), (fa_u32)(gn & 1), abort_flag);
        // the first products of an item overwrite dV and dK: the drain warps must have read the
        // previous item's out of TMEM
        if (ok && n == 0 && kvc > 0) ok = fa_mbar_wait_all(bar_addr(sb, BAR_DKVFREE), (fa_u32)((kvc - 1) & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        // B operands read MN-major: the D columns are 64-element groups TILE_BYTES apart, a
        // k-step is 16 q rows = 2048 bytes
        const fa_u32 loQ_mn = fa_desc_lo(sb + OFF_Q + s * TILE_BYTES, TILE_BYTES);
        const fa_u32 loDO_mn = fa_desc_lo(sb + OFF_DO + s * TILE_BYTES, TILE_BYTES);
        const fa_u32 loDS_k = fa_desc_lo(sb + OFF_DS + (gn % NDS) * DS_BYTES, 16);
        const fa_u32 acc = n > 0;  // the first pair of an item starts its dK and dV
        // 3. dV += P^T dO      (K = BQ q values; A from TMEM)
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk)
          if (leader) fa_mma_ts(tmem_u + COL_DV, tmem_u + COL_P + kk * 8, fa_desc_make(loDO_mn + kk * 128, HI), IDESC_TN, acc | (kk > 0));
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_DOEMPTY + s));  // second arrival: the dO tile is free
          // two dS^T buffers: P^T is free, and so is the other buffer (product 4 of the previous pair came before)
          if (NDS == 2) fa_mma_commit(bar_addr(sb, BAR_PFREE));
        }
        // 4. dK += dS^T Q     (A = dS^T K-major: k-step kk is 32 bytes into atom kk / 4)
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk)
          if (leader)
            fa_mma_ss(tmem_u + COL_DK, fa_desc_make(loDS_k + kstep_kmajor(kk, TILE_BYTES), HI),
                      fa_desc_make(loQ_mn + kk * 128, HI), IDESC_TN, acc | (kk > 0));
        if (leader) {
          fa_mma_commit(bar_addr(sb, BAR_QEMPTY + s));   // second arrival: the Q tile and row scalars are free
          if (NDS == 1) fa_mma_commit(bar_addr(sb, BAR_PFREE));  // one of the two arrivals that free P^T and dS^T
          if (n + 1 == np) fa_mma_commit(bar_addr(sb, BAR_FINAL + kvc % KVBUF));
        }
      }
      ++kvc;
    }
  } else if (warp == WARP_MMA_C) {
    // ================================ MMA issuer C: product 5 ==================================
    // (a third issuing warp: what bounds the tensor core in this kernel is how fast one thread
    //  can issue, so the instructions of a pair are spread over three threads)
    const bool leader = fa_elect_one();
    constexpr fa_u32 IDESC_NN = fa_idesc(DT, 128, 64, 1, 1);    // A, B MN-major, M = 128, N = 64
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    bool ok = true;
    int gn = 0, kvc = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int np = __shfl_sync(0xffffffffu, item[4 * lb + 3], 0);
      if (leader) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
      if (np < 0) break;
      if (np == 0) continue;
      const int kb = kvc % KVBUF;
      const fa_u32 loK_mn = fa_desc_lo(sb + OFF_K + kb * TILE_BYTES, TILE_BYTES);
      ok = fa_mbar_wait_all(bar_addr(sb, BAR_KV + kb), (fa_u32)((kvc / KVBUF) & 1), abort_flag);
      for (int n = 0; n < np && ok; ++n, ++gn) {
        ok = fa_mbar_wait_all(bar_addr(sb, BAR_PREADY), (fa_u32)(gn & 1), abort_flag);
        if (NDS == 2 && ok && leader) {
          // product 5 of the previous pair is the last reader of the other dS^T buffer
          if (gn > 0) fa_mma_commit(bar_addr(sb, BAR_PFREE));
          else fa_mbar_arrive(bar_addr(sb, BAR_PFREE));
        }
        // the drain warps must have emptied the dQ columns of the previous pair
        if (ok && gn > 0) ok = fa_mbar_wait_all(bar_addr(sb, BAR_DQFREE), (fa_u32)((gn - 1) & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        const fa_u32 loDS_mn = fa_desc_lo(sb + OFF_DS + (gn % NDS) * DS_BYTES, TILE_BYTES);
        // 5. dQ = dS K: K = 128 kv rows, a k-step is 16 rows = 2048 bytes of either operand; A = dS^T read MN-major
        //    (M = 128 q: two 64-column atoms), B = K (N = 64 d)
#pragma unroll
        for (int kk = 0; kk < BT / 16; ++kk)
          if (leader) fa_mma_ss(tmem_u + COL_DQ, fa_desc_make(loDS_mn + kk * 128, HI), fa_desc_make(loK_mn + kk * 128, HI), IDESC_NN, kk > 0);
        if (leader) {
          if (NDS == 1) fa_mma_commit(bar_addr(sb, BAR_PFREE));
          fa_mma_commit(bar_addr(sb, BAR_DQFULL));
          if (n + 1 == np) fa_mma_commit(bar_addr(sb, BAR_FINAL + kb));  // (this product is the last reader of K)
        }
      }
      ++kvc;
    }
  } else if (warp < 8) {
    // ================================ compute warps ============================================
    fa_setmaxnreg_inc<REGS_COMPUTE>();
    const int half = warp >> 2;               // q columns CW*half .. +CW-1 of the pair tile
    const int lane_base = (warp & 3) * 32;
    const int r = lane_base + lane;           // kv row of this thread inside the tile
    const fa_u32 t_row = tmem + ((fa_u32)lane_base << 16);
    const float sc2 = p.scale * FA_LOG2E;
    bool ok = true;
    int gn = 0;
    for (int itc = 0; ok; ++itc) {
      const int lb = itc & 1;
      ok = fa_mbar_wait_warp(bar_addr(sb, BAR_LISTFULL + lb), (fa_u32)((itc >> 1) & 1), abort_flag);
      if (!ok) break;
      const int idx = KVBUF == 2 ? item[4 * lb] : 0, np = item[4 * lb + 3];
      if (np < 0) break;
      const int* pl = pairs + lb * MAXPL;
      const Item it = read_item(idx, item + 4 * lb, p.Hkv, p.B);
      const int hk = it.hk, b = it.b, n0 = it.kt * BT;
      const int gb = b + p.b_off;
      const int kv = n0 + r;
      const bool row_ok = kv < p.Skv;
      const unsigned* bits = bits_row(p, kv);
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int s = gn % NSTAGE;
        const int pr = pl[n];
        const int m0 = (pr & 0xffff) * BQ, h = hk * G + (pr >> 20), gh = h + p.h_off;
        bool masked = FA_HAS_MASK_MOD && ((pr >> 16) & 0xf) == 1;
        // the mask of this thread's 64 columns, read (where it was evaluated beforehand: while S^T is waited for) or evaluated.  (Asked
        // for a pair ahead, as at head dim 128, the words cost more registers than they save: packed documents 97 -> 99 us.)
        fa_u32 keep[2];
        keep[0] = keep[1] = 0xffffffffu;
        if (masked && row_ok) {
          if (bits != nullptr) read_keep(keep, bits, p, b, h, m0 + half * CW);
          else eval_keep(keep, gb, gh, m0 + half * CW, kv);
        }
        masked |= clear_beyond(keep, p.Sq - (m0 + half * CW));
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_SFULL), (fa_u32)(gn & 1), abort_flag);
        if (ok) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_QFULL + s), (fa_u32)((gn / NSTAGE) & 1), abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        const float* rowp = (const float*)(sm + OFF_ROW + s * 2 * BQ * 4);
        fa_u32 pp[CW / 2], ds[CW / 2];
        // The CW columns of this thread come in steps of 16 (S^T and dP^T), the loads of a step in
        // flight while the previous one is computed: few values are live at a time, which leaves
        // the scheduler registers to overlap the latencies of independent elements (with all the
        // values loaded up front this loop ran at 28 clocks per element).
        {
          const fa_u32 tS = t_row + COL_S + half * CW, tD = t_row + COL_DP + half * CW;
          const int c0 = half * CW;  // first q column of this thread inside the tile
          float sA[16], dA[16], sB[16], dB[16];
          fa_u32 p8[8], d8[8];
          fa_tmem_ld16(tS, sA);
          fa_tmem_ld16(tD, dA);
          fa_tmem_wait_ld();
#define FA_STEP(SC, DC, SN, DN, C, LAST)                                                                   \
  if (!(LAST)) {                                                                                           \
    fa_tmem_ld16(tS + (C) + 16, SN);                                                                       \
    fa_tmem_ld16(tD + (C) + 16, DN);                                                                       \
  } else {                                                                                                 \
    /* every score of the pair is in registers: the S^T / dP^T columns may be overwritten */              \
    fa_tc_fence_before();                                                                                  \
    fa_mbar_arrive(bar_addr(sb, BAR_SFREE));                                                               \
  }                                                                                                        \
  if (row_ok) {                                                                                            \
    chunk<16>(SC, DC, rowp + c0 + (C), rowp + BQ + c0 + (C), p8, d8, m0 + c0 + (C), kv, gb, gh, p.scale, sc2); \
  } else {                                                                                                 \
    _Pragma("unroll") for (int e = 0; e < 8; ++e) p8[e] = d8[e] = 0u;                                      \
  }                                                                                                        \
  _Pragma("unroll") for (int e = 0; e < 8; ++e) {                                                          \
    pp[(C) / 2 + e] = p8[e];                                                                               \
    ds[(C) / 2 + e] = d8[e];                                                                               \
  }                                                                                                        \
  if (!(LAST)) fa_tmem_wait_ld();
          FA_STEP(sA, dA, sB, dB, 0, false)
          FA_STEP(sB, dB, sA, dA, 16, false)
          FA_STEP(sA, dA, sB, dB, 32, false)
          FA_STEP(sB, dB, sA, dA, 48, true)
#undef FA_STEP
        }
        // pin the packed results here: without this the compiler sinks part of the math below the
        // wait that follows, onto the critical path between two groups of products
#pragma unroll
        for (int e = 0; e < CW / 2; ++e) asm volatile("" : "+r"(pp[e]), "+r"(ds[e]));
        if (masked) {
          mask_pairs(pp, ds, keep[0]);
          mask_pairs(pp + 16, ds + 16, keep[1]);
        }
        // product 3 of the previous pair must be done with P^T, and products 4-5 of the last pair that used this
        // dS^T buffer with that
        if (gn > 0) {
          ok = fa_mbar_wait_warp(bar_addr(sb, BAR_PFREE), (fa_u32)((gn - 1) & 1), abort_flag);
          if (!ok) break;
          fa_tc_fence_after();
        }
#pragma unroll
        for (int i = 0; i < CW / 32; ++i)
          fa_tmem_st16(t_row + COL_P + half * (CW / 2) + 16 * i, *(const fa_u32(*)[16])(pp + 16 * i));
        {
          // dS^T row r: this thread's CW columns are CW / 8 sixteen-byte chunks; chunk ck of a 128-byte
          // atom row goes to position ck ^ (r & 7) (the 128-byte swizzle of the operand layout)
#pragma unroll
          for (int c = 0; c < CW / 8; ++c) {
            const int col = half * CW + 8 * c;
            unsigned char* dsrow = sm + OFF_DS + (gn % NDS) * DS_BYTES + (col >> 6) * TILE_BYTES + r * 128;
            uint4 w;
            w.x = ds[4 * c]; w.y = ds[4 * c + 1]; w.z = ds[4 * c + 2]; w.w = ds[4 * c + 3];
            *(uint4*)(dsrow + ((((col & 63) >> 3) ^ (r & 7)) * 16)) = w;
          }
        }
        fa_tmem_wait_st();
        fence_proxy_async();
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_PREADY));
      }
      if (!ok) break;
      // every lane has read its last list entry: the list may be overwritten
      __syncwarp();
      if (lane == 0) fa_mbar_arrive(bar_addr(sb, BAR_LISTFREE + lb));
    }
  } else if (warp < 12) {
    // ================================ drain warps: dQ of every pair, dK / dV of every item =======
    const int lane_base = (warp & 3) * 32;
    const int r = lane_base + lane;  // TMEM lane: q row of the pair; kv row for dK / dV
    const fa_u32 t_lane = tmem + ((fa_u32)lane_base << 16);
    const fa_u32 t_dq = t_lane + COL_DQ;
    const int dtid = tid - 256;
    const int n_qtiles = sq_pad / BQ;
    unsigned char* const dqrow = sm + OFF_DQ + r * 128;  // this thread's row of the staging buffer
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
      const int idx = KVBUF == 2 ? item[4 * lb] : 0, np = item[4 * lb + 3];
      if (np < 0) break;  // (the same in all four warps)
      const int* pl = pairs + lb * MAXPL;
      const Item it = read_item(idx, item + 4 * lb, p.Hkv, p.B);
      const int hk = it.hk, b = it.b, n0 = it.kt * BT;
      for (int n = 0; n < np && ok; ++n, ++gn) {
        const int pr = pl[n];
        const int qt = pr & 0xffff, h = hk * G + (pr >> 20);
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_DQFULL), (fa_u32)(gn & 1), abort_flag);
        fa_tc_fence_after();
        if (!ok) break;
        // The whole row comes into registers, so that the columns are free at once; it leaves by 32 columns through the
        // warp's own 4 KB of staging, each time one bulk reduce-add of 4 KB (no barrier between the warps).  16-byte chunk k of
        // lane r goes to position k ^ (r & 7), which spreads the rows over the banks.
        float* gdst = P.dq_acc + (((long long)b * p.Hq + h) * n_qtiles + qt) * (128 * D) + (warp & 3) * 1024;
        float a[2][32];
        fa_tmem_ld32(t_dq, a[0]);
        fa_tmem_ld32(t_dq + 32, a[1]);
        fa_tmem_wait_ld();
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_DQFREE));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (lane == 0) bulk_wait_read0();  // the previous reduce (or store) has read the staging buffer
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            *(float4*)(dqrow + ((k ^ (r & 7)) * 16)) = make_float4(a[c][4 * k], a[c][4 * k + 1], a[c][4 * k + 2], a[c][4 * k + 3]);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            bulk_reduce_add_f32(gdst + c * 4096, sb + OFF_DQ + (warp & 3) * 4096, 4096);
            bulk_commit();
          }
        }
      }
      // ---- dK (scaled) and dV of the item.  A thread owns one kv row (TMEM lane); 64 columns at a
      // time are converted into the staging buffer in the layout of a K tile (128-byte rows, 16-byte
      // chunk k of row r at k ^ (r & 7)) and leave through one tensor-map store, which writes whole
      // lines and clips the rows beyond Skv.  (Each thread storing its own row straight to global
      // memory took several thousand cycles per item: 32 different lines per instruction.)
      // An item without pairs has zeros written.
      if (np > 0) {
        const int kb = kvc % KVBUF;
        if (ok) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_FINAL + kb), (fa_u32)((kvc / KVBUF) & 1), abort_flag);
        if (!ok) misc[3] = 1;
        named_bar_sync(1, 128);
        if (misc[3] != 0) {
          ok = false;
          break;
        }
        fa_tc_fence_after();
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {  // dK, dV
          const float mul = which == 0 ? p.scale : 1.f;
          // two K / V buffers: the staging buffers are the item's own K and V tiles, which nothing reads
          // any more; one: the parts go through the dQ staging buffer one after the other
          const int st_off = KVBUF == 2 ? (which == 0 ? OFF_K : OFF_V) + kb * TILE_BYTES : OFF_DQ;
          unsigned char* strow = sm + st_off + r * 128;
          if (KVBUF == 1) {
            // the previous bulk operations must have finished reading the staging buffer
            if (lane == 0) bulk_wait_read0();
            named_bar_sync(1, 128);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float o[16];
            fa_tmem_ld16(t_lane + (which == 0 ? COL_DK : COL_DV) + c * 16, o);
            fa_tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; e += 8) {
              uint4 w;
              w.x = fa_pack2<DT>(o[e] * mul, o[e + 1] * mul);
              w.y = fa_pack2<DT>(o[e + 2] * mul, o[e + 3] * mul);
              w.z = fa_pack2<DT>(o[e + 4] * mul, o[e + 5] * mul);
              w.w = fa_pack2<DT>(o[e + 6] * mul, o[e + 7] * mul);
              *(uint4*)(strow + (((2 * c + (e >> 3)) ^ (r & 7)) * 16)) = w;
            }
          }
          if (which == 1) {
            // dK and dV are out of TMEM: the next item's first products may overwrite them
            fa_tc_fence_before();
            fa_mbar_arrive(bar_addr(sb, BAR_DKVFREE));
          }
          if (KVBUF == 1 || which == 1) {
            fence_proxy_async();
            named_bar_sync(1, 128);
          }
          if (dtid == 0) {
            if (KVBUF == 1) {
              fa_tma_store_4d(which == 0 ? &P.tdk : &P.tdv, sb + OFF_DQ, 0, n0, hk, b);
              bulk_commit();
            } else if (which == 1) {
              fa_tma_store_4d(&P.tdk, sb + OFF_K + kb * TILE_BYTES, 0, n0, hk, b);
              fa_tma_store_4d(&P.tdv, sb + OFF_V + kb * TILE_BYTES, 0, n0, hk, b);
              bulk_commit();
              bulk_wait_read0();
              fa_mbar_arrive(bar_addr(sb, BAR_KVFREE + kb));
            }
          }
        }
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
      if (np > 0) {
        if (KVBUF == 1) {  // (the staging buffer is the warps' own again once the last store has read it)
          if (dtid == 0) bulk_wait_read0();
          named_bar_sync(1, 128);
        }
        ++kvc;
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
