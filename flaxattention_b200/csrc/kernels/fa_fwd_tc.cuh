// Flash-attention forward for sm_100a on the 5th-generation tensor cores:
//   S = Q K^T and O += P V are tcgen05.mma instructions with accumulators in TMEM,
//   Q / K / V tiles arrive by TMA (128-byte swizzle) through an mbarrier ring,
//   the softmax runs thread-per-row on scores read once from TMEM into registers, and P goes
//   back to TMEM as 16-bit pairs to be the A operand of the second product (its own columns
//   with D = 64, over the score columns with D = 128).
// Same math and BlockMask walk as fa_fwd.cuh (see there for the reference citations); this
// kernel covers fp16 / bf16, D = Dv in {64, 128}, block sizes that are multiples of 128 and a
// positive scale; and fp32, D = Dv = 64, in the form described next.
//
// fp32 (FA_DTYPE 2).  The tensor cores multiply no fp32 operands without dropping mantissa bits, so
// every operand is written as a sum of three bf16 values, hi + mid + lo, which holds all 24 mantissa bits
// (each part is the rounding of what the parts before it leave; bf16 has the exponent range of fp32):
// q, k and v by a small kernel in front of this one, whose rows are [hi | mid | lo] (192 values), and the
// probabilities by the softmax threads.  A product is then the six bf16 products hi.hi, hi.mid,
// mid.hi, mid.mid, hi.lo, lo.hi, accumulated in fp32, smallest first; the three left out are below
// 2^-25 of hi.hi, half a unit in the last place of an fp32 product.  The tensor core adds into its fp32
// accumulator without rounding to nearest, so nothing is accumulated there for long: the P.V product
// of every kv step starts from zero and the softmax threads add it to the output row they keep in
// registers (with O accumulated in TMEM over all steps the error grew to five times that of the FMA
// kernel at 1024 keys).  The softmax keeps the operations and their order of fa_fwd.cuh.  Error against 64 bits
// (2-norm of the difference over that of the output): 1.7e-7 to 3.7e-7 where the FMA kernel has 3.3e-7 to 1.2e-6
// (97 to 4096 keys).  Infinities, NaN and |x| >= 2^30 have no parts that give the right result (inf - inf, 0 * inf, sums
// that leave the range): the split kernel notes them, and fa_fwd_rerun_kernel does those heads over.
//
// One CTA owns two 128-row query tiles of one (batch, head) and streams 128-row K/V tiles
// past both (or one, see NQ: then without warps 4-7, and the roles below move up).  Warp roles (12 warps = 3 warpgroups):
//   warps 0-3  softmax warpgroup of query tile 0      warps 4-7  of query tile 1
//   warp 8     TMA producer (one lane)
//   warps 9-10 MMA issuers; warp 9 also allocates / frees TMEM.  With D = 64 each issues the products of one query tile;
//              where P lies over S for the rest of the step (D = 128, fp32) warp 9 issues all products of both query
//              tiles in turn; in the decode variant warp 9 issues the S products and warp 10 the PV products.  Warp 11 is idle
// Registers are moved from the third warpgroup to the two softmax warpgroups (setmaxnreg),
// which hold a whole 128-column score row per thread.
// With D = 64 the S columns of a tile are released as soon as its scores are in registers, and S of step j+1 is
// computed while the softmax of step j runs (see ROT); with D = 128 (P over the S columns) the products of a tile form
// the chain  PV(j), S(j+1), PV(j+1) ... and all the latencies between them count: P is handed over in two parts (see
// SPLIT_P), and the issuing warp has waited for everything else that a product needs before P is there.
// What bounds it (clock stamps, dense, two tiles): D = 64, a step of both tiles is 2400 clk, of which 2060 are the
// instructions of the two softmax warps of a scheduler (two warps in a loop of their own, without barriers and
// products, take that; the SFU alone 1536); D = 128, 2900 clk of chain against 2048 clk of products.  B8 H8 S2048 D64
// checkerboard 124 -> 116 us, B4 H8 S4096 D64 208 -> 198, D128 267 -> 258, attention sink B4 H16 S8192 D128 411 -> 363.
// The running maximum is only raised when it grew by more than 2^8 (the stale maximum is
// exact as long as it is used consistently), so rescaling O in TMEM is rare.
//
// Every mbarrier wait is bounded; on expiry the CTA raises FA_STATUS_WAIT_TIMEOUT in the
// status word, all roles leave their loops, TMEM is freed and the kernel returns.
//
// Compile-time parameters (macros): FA_DTYPE (0 fp16, 1 bf16, 2 fp32), FA_D (64 or 128), FA_TC_DECODE
// (split-KV variant, see below), FA_TC_NQ (query tiles of a CTA, see below).
#pragma once
#include "fa_sm100.cuh"

struct FaTcParams {
  FaParams p;
  FaTensorMap tq, tk, tv;  // 4-d maps (D, S, H, B), box 64 x 128 x 1 x 1, 128-byte swizzle
  FaTensorMap to;          // the output, like tq (unused by the decode variant, which writes partial results)
};

namespace fa_tc {

constexpr bool F32 = FA_DTYPE == FA_DT_F32;
constexpr int DT = F32 ? FA_DT_BF16 : FA_DTYPE;  // type of the tensor-core operands
constexpr int D = FA_D;
constexpr int BM = 128, BN = 128;
constexpr int NPART = F32 ? 3 : 1;       // bf16 parts of an operand value
constexpr int ATOMS = NPART * D / 64;    // 64-element (128-byte) column groups per row (fp32: one per part)
constexpr int ATOM_BYTES = 128 * 128;    // 128 rows x 128 bytes
// Split-KV decode variant (FA_TC_DECODE, D = 64, at most 64 query rows): the CTA owns a contiguous
// share of the kv tiles the BlockMask lists and the two softmax warpgroups take alternate kv tiles
// of that share.  A warpgroup's 128-row tile holds the query rows twice, in rows 0-63 and again in
// rows 64-127, so that two threads work on one query row: the thread of TMEM lane r < 64 takes kv
// columns 0-63 of the tile, the thread of lane r + 64 columns 64-127.  Each thread runs its own
// online softmax over its half tiles (own running maximum and sum) and writes P for its columns
// only; the other 64 columns of its lane are zero, so the P.V product gives every lane the
// partial output of its own columns.  No thread sits on a padding row while there are at least
// 33 queries, and a thread's serial work per kv tile is half that of the forward.  At the end the
// four partial results of a row (running maximum, sum, O of two warpgroups x two halves) are
// merged through shared memory and the CTA writes one un-normalised partial result per row for
// the combine kernel.  More stages, since the kv stream is all there is.
#ifndef FA_TC_DECODE
#define FA_TC_DECODE 0
#endif
constexpr bool DECODE = FA_TC_DECODE != 0;
// (fp32: the parts of two query tiles, a K and a V tile fill shared memory; K of the next step is loaded
// during the softmax and the PV products of this one, V during the next S products)
// Query tiles of a CTA (decode: copies of the query tile).  One (FA_TC_NQ 1): two CTAs share an SM, so that the
// set-up, first loads and epilogue of one run under the steps of the other and the last wave of the grid is
// finer; K and V are then loaded for every query tile, through a shorter ring.  The host picks.
#ifndef FA_TC_NQ
#define FA_TC_NQ 2
#endif
constexpr int NQ = FA_TC_NQ;
static_assert(NQ == 2 || (NQ == 1 && !DECODE && !F32), "one query tile: 16-bit forward");
constexpr int NSTAGE = DECODE ? 5 : (F32 ? 1 : (D == 64 ? NQ + 1 : NQ));
constexpr int Q_BYTES = NQ * ATOMS * ATOM_BYTES;
constexpr int KV_STAGE = ATOMS * ATOM_BYTES;
constexpr int MAXT = 256;                // kv tiles per row of the block grid (Skv <= 32768)
constexpr int NBARS = 1 + 4 * NSTAGE + 13;
constexpr int OFF_K = Q_BYTES;
constexpr int OFF_V = OFF_K + NSTAGE * KV_STAGE;
constexpr int OFF_BAR = OFF_V + NSTAGE * KV_STAGE;
constexpr int OFF_MISC = OFF_BAR + NBARS * 8;       // tmem base, abort flag, nsteps, pad
constexpr int OFF_SCHED = OFF_MISC + 16;            // u32 sched[MAXT + 4]: kv tile | mode of query tile 0 << 16 | mode of query tile 1 << 24
constexpr int OFF_CLS = OFF_SCHED + (MAXT + 4) * 4; // uchar cls[2][MAXT]
constexpr int OFF_WCNT = OFF_CLS + 2 * MAXT;        // int wcount[MAXT / 32]: listed tiles per warp of the schedule build
constexpr int SMEM_BYTES = OFF_WCNT + (MAXT / 32) * 4 + 1024;  // + slack for the 1024-byte alignment
constexpr int TMEM_COLS = 256 * NQ;
// fp32: scores of tile i in columns 192 i .. + 127.  The softmax writes the parts of P over the scores it
// has just read, 16 columns (32 keys) at a time: hi and mid of keys 32 c .. + 31 go to columns 32 c .. + 15
// and 32 c + 16 .. + 31, lo to 128 + 16 c .. + 15.  O of tile i and step in 384 + 64 i.
// Head dim 64, forward (ROT): each tile has 192 columns for S and P.  In even steps S takes columns 0-127 and P
// goes over columns 0-63, in odd steps S takes columns 64-191 and P goes over columns 128-191.  S of the next step
// then never lies over P of this one (it is computed during this step's softmax), and P of a step never lies over
// P of the last one, so the softmax does not wait for any P.V product.
constexpr bool ROT = D == 64 && !F32 && !DECODE;
constexpr int COL_S = 0, COL_O = F32 ? 384 : (ROT ? 192 : 128) * NQ, S_STRIDE = F32 || ROT ? 192 : 128;
// In the decode variant P has columns of its own (384..511).  With D = 128 the 512 columns are taken by S and O, and
// P overwrites the S columns it was computed from.
constexpr int COL_P = 192 * NQ;
// One pair of exponentials in FA_TC_POLY_EVERY goes to the FMA pipe (a cubic, see fa_ex2_poly2).
// Measured (B8 H8 S2048 D64): every fourth pair takes the forward without a score_mod from 0.118 to
// 0.114 ms, with the checkerboard mod from 0.133 to 0.129 and causal + ALiBi from 0.088 to 0.085;
// every eighth is about the same, every third and every second are slower again (the issue slots).
// The same for one and for two query tiles per CTA: which of the two a call gets depends on its batch size and on a hint,
// and its results must not.  (Every fifth with two tiles and no score_mod takes D64 B2 H8 S8192 causal from 193 to 188 us, D128 B2 H16/4
// S3001 from 90.9 to 88.8, but then the rows of a shard differ from those of the whole.)
#ifndef FA_TC_POLY_EVERY
#define FA_TC_POLY_EVERY 4
#endif
constexpr int NSOFT = 4 * NQ;           // softmax warps
constexpr int NT = (NSOFT + 4) * 32;
// Register split (setmaxnreg): a thread starts with 168 registers with two query tiles (65536 / 384, rounded
// down to a multiple of 8) and with 128 with one (two CTAs of 256 threads on an SM).  The last warpgroup gives
// some up and the softmax warpgroups take them.  The increase must not ask for more than the
// decrease releases: setmaxnreg.inc blocks until the registers are there, without a time limit.
constexpr int REGS_LAUNCH = NQ == 2 ? 168 : 128, REGS_SOFTMAX = NQ == 2 ? 200 : 192, REGS_OTHER = NQ == 2 ? 96 : 64;
static_assert(NQ * (REGS_SOFTMAX - REGS_LAUNCH) <= REGS_LAUNCH - REGS_OTHER, "setmaxnreg.inc would wait forever");
constexpr int WARP_PRODUCER = NSOFT, WARP_MMA = NSOFT + 1, WARP_MMA_B = NSOFT + 2;
constexpr float RESCALE_THRESHOLD = 8.0f;  // log2 units
constexpr float REL_FLOOR = -64.0f;         // log2 units

static_assert(D == 64 || D == 128, "head dim 64 or 128");
static_assert(!DECODE || D == 64, "the decode variant is written for head dim 64");
static_assert(!F32 || (D == 64 && !DECODE), "fp32: head dim 64, forward");
// the pairs of parts whose products are kept, smallest first
constexpr int NPROD = F32 ? 6 : 1;
__device__ constexpr int PROD_A[6] = {F32 ? 1 : 0, 0, 2, 0, 1, 0}, PROD_B[6] = {F32 ? 1 : 0, 2, 0, 1, 0, 0};

__device__ __forceinline__ fa_u32 bar_addr(fa_u32 sbase, int i) { return sbase + OFF_BAR + i * 8; }
constexpr int BAR_Q = 0;
constexpr int BAR_KFULL = 1, BAR_KEMPTY = 1 + NSTAGE, BAR_VFULL = 1 + 2 * NSTAGE, BAR_VEMPTY = 1 + 3 * NSTAGE;
// ROT: two barriers per tile for P and O, BAR_P + i and BAR_O + i for even steps, + 2 for odd ones.  (The warps of a
// tile only meet at its S: one that is ahead may hand over P of a step before the others have handed over that of
// the last one, and the softmax does not look at every PV product.)
constexpr int BAR_S = 1 + 4 * NSTAGE, BAR_P = BAR_S + 2, BAR_O = BAR_S + 6;
// Where P does not lie over S of the same step for long (ROT, DECODE), the S columns of a tile are released as soon as
// the softmax warps hold the scores in registers, and S of the next step is produced during the softmax.
constexpr int BAR_SFREE2 = BAR_S + 10;
constexpr int BAR_LAG = BAR_S + 12;  // (ROT) the first PV product of the second tile is complete; used once
constexpr bool EARLY_S = ROT || DECODE;
// Head dim 128: P is handed over in two parts, keys 0-95 (BAR_P) and 96-127 (BAR_P2), so that most of the PV product
// runs under the last exponentials.  It is the first link of the chain PV(j), S(j+1) that the tile then waits for.
constexpr bool SPLIT_P = !ROT && !DECODE && !F32;
constexpr int BAR_P2 = BAR_S + 10;

// Work on one 32-column chunk of a score row held in registers (columns C0 .. C0+31 of the kv
// tile that starts at key n0).  C0 is a template parameter and n0 a multiple of 128, so the low
// bits of every key index are compile-time constants inside the mods.
struct RowMax {
  float a, b, c, d;
};
__device__ __forceinline__ void max_chunk(const float (&v)[32], RowMax& mx) {
#pragma unroll
  for (int e = 0; e < 32; e += 8) {
    mx.a = fa_max3(mx.a, v[e], v[e + 1]);
    mx.b = fa_max3(mx.b, v[e + 2], v[e + 3]);
    mx.c = fa_max3(mx.c, v[e + 4], v[e + 5]);
    mx.d = fa_max3(mx.d, v[e + 6], v[e + 7]);
  }
}
// score_mod (and the rounding of the raw scores to the input type, when asked for) in place.  With a score_mod the
// results are in log2 units and relative to the row's running maximum (negm is added; not where that is far below 0, see
// m_base): where that does not move, the exponentials are taken of them as they are, without a subtraction of their own.  An affine score_mod
// (A * score + B) costs one packed FMA per pair: A and B absorb the scale, log2(e) and the maximum.
// (Without a score_mod the scores stay raw, the exponent's FMA applies the scale.)
struct ModLinear {
  fa_u64 m2, od[4];  // multiplier; 0 and 1, 2 and 3, 4 and 5, 6 and 7 times the slope over kv
  float d, b;        // slope; bias at the first key of the tile (with the maximum)
};
template <int C0>
__device__ __forceinline__ void mod_chunk(float (&v)[32], int n0, int qi, int gb, int gh, float scale, float sc2, float negm,
                                          const ModLinear& lin) {
  [[maybe_unused]] float at8 = 0.f;
#pragma unroll
  for (int e = 0; e < 32; e += 2) {
    float x0 = v[e], x1 = v[e + 1];
    [[maybe_unused]] const int kv0 = n0 | (C0 + e), kv1 = n0 | (C0 + e + 1);
#if FA_ROUND_SCORES
    fa_round2<DT>(x0, x1);
#endif
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE) && defined(FA_SCORE_LINEAR_KV)
    // The multiplier does not read kv and the bias is linear in it (relative-position biases such as ALiBi): both are
    // taken once per step, at the first key of the tile; every eighth column is reached from there with one FMA and the
    // columns behind it with an addition, both packed - instead of an integer subtraction, an int-to-float conversion
    // (which shares the SFU with the exponentials) and a multiplication per element.  (A packed FMA per pair with the column
    // numbers as constants needs those in registers, two moves per pair: B2 H1 S8192, D64 rounded 103 us against 99, D128 104 against 103,
    // causal D64 88 against 82.)
    if (e % 8 == 0) at8 = fmaf((float)(C0 + e), lin.d, lin.b);
    fa_f2_unpack(fa_fma2(fa_f2(x0, x1), lin.m2, fa_add2(fa_f2(at8, at8), lin.od[(e % 8) / 2])), x0, x1);
#elif FA_HAS_SCORE_MOD && defined(FA_SCORE_MUL_ONLY)
    fa_f2_unpack(fa_fma2(fa_f2(x0, x1), fa_f2(fa_score_mul(0.f, gb, gh, qi, kv0) * sc2, fa_score_mul(0.f, gb, gh, qi, kv1) * sc2), fa_f2(negm, negm)), x0, x1);
#elif FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE)
    fa_f2_unpack(fa_fma2(fa_f2(x0, x1), fa_f2(fa_score_mul(0.f, gb, gh, qi, kv0) * sc2, fa_score_mul(0.f, gb, gh, qi, kv1) * sc2),
                         fa_add2(fa_f2(fa_score_add2(0.f, gb, gh, qi, kv0), fa_score_add2(0.f, gb, gh, qi, kv1)), fa_f2(negm, negm))), x0, x1);
#elif FA_HAS_SCORE_MOD
    x0 = fmaf(fa_score_mod(x0 * scale, gb, gh, qi, kv0), FA_LOG2E, negm);
    x1 = fmaf(fa_score_mod(x1 * scale, gb, gh, qi, kv1), FA_LOG2E, negm);
#endif
    v[e] = x0;
    v[e + 1] = x1;
  }
}
// mask_mod (on tiles the BlockMask lists as partial) and the end of the sequence (ragged last
// tile): masked scores become -inf.  Only the few tiles that need it come here, so the code is
// kept small rather than fast: a rolled loop evaluates the mask of this thread's columns into
// one word per 32 columns, and the words are applied to the registers.  (A second copy of the whole step with the
// mask evaluated in line, per element and fully unrolled, made a masked step take 12-15k clocks
// against 3.5k for a plain one: the step no longer fitted the instruction cache.)
template <int NW>
__device__ __forceinline__ void mask_bits(fa_u32 (&w)[NW], bool use_mask, int kv0, int qi, int gb, int gh, int Skv,
                                          bool have_words, const uint4& m) {
  // the end of the sequence alone needs no loop: word c covers keys kv0 + 32 c .. + 31
#pragma unroll
  for (int c = 0; c < NW; ++c) {
    const int left = Skv - (kv0 + 32 * c);
    w[c] = left >= 32 ? 0xffffffffu : (left <= 0 ? 0u : ((1u << left) - 1u));
  }
#if FA_HAS_MASK_MOD
  if (use_mask && have_words) {
    // mask_mod was evaluated once for all positions (FaTables::mask_bits): this row's words of the tile
    w[0] &= m.x; w[1] &= m.y;
    if (NW == 4) { w[NW > 2 ? 2 : 0] &= m.z; w[NW > 2 ? 3 : 0] &= m.w; }
  } else if (use_mask) {
    // one rolled loop, the NW words side by side (independent evaluations in every iteration)
    fa_u32 m[NW];
#pragma unroll
    for (int c = 0; c < NW; ++c) m[c] = 0u;
#pragma unroll 2
    for (int e = 0; e < 32; ++e) {
#pragma unroll
      for (int c = 0; c < NW; ++c) m[c] |= (fa_mask_mod(gb, gh, qi, kv0 + 32 * c + e) ? 1u : 0u) << e;
    }
#pragma unroll
    for (int c = 0; c < NW; ++c) w[c] &= m[c];
  }
#endif
}
// the words of a row of the bit matrix for the NW * 32 keys from kv0 on
template <int NW>
__device__ __forceinline__ uint4 mask_words(const unsigned* rowbits, int kv0) {
  if (NW == 4) return *(const uint4*)(rowbits + (kv0 >> 5));
  const uint2 m = *(const uint2*)(rowbits + (kv0 >> 5));
  return make_uint4(m.x, m.y, 0u, 0u);
}
__device__ __forceinline__ void mask_apply(float (&v)[32], fa_u32 bits) {
#pragma unroll
  for (int e = 0; e < 32; ++e) v[e] = ((bits >> e) & 1u) ? v[e] : FA_NEG_INF;
}

// Pass-2 work on one chunk: p = 2^(x * cmul - m) (REL: 2^x, the scores are relative to m already), packed to 16 bits,
// and the row-sum chains.
template <bool REL, int E0, int E1>
__device__ __forceinline__ void pass2_part(const float (&v)[32], fa_u32 (&pk)[16], fa_u64 cmul, fa_u64 negm,
                                           fa_u64& sum_a, fa_u64& sum_b) {
#pragma unroll
  for (int e = E0; e < E1; ++e) {
    float a0 = v[2 * e], a1 = v[2 * e + 1];
    if (!REL) fa_f2_unpack(fa_fma2(fa_f2(a0, a1), cmul, negm), a0, a1);
    // one pair in FA_TC_POLY_EVERY takes its exponentials on the FMA pipe: the SFU (16 per clock
    // and SM) is what bounds this loop
    float p0, p1;
    if (FA_TC_POLY_EVERY > 0 && (e % (FA_TC_POLY_EVERY > 0 ? FA_TC_POLY_EVERY : 1)) == (FA_TC_POLY_EVERY - 1)) {
      fa_ex2_poly2(a0, a1, p0, p1);
    } else {
      p0 = fa_ex2(a0);
      p1 = fa_ex2(a1);
    }
    pk[e] = fa_pack2<DT>(p0, p1);
    const fa_u64 pf = fa_f2(p0, p1);
    if (e & 1) sum_b = fa_add2(sum_b, pf);
    else sum_a = fa_add2(sum_a, pf);
  }
}

template <bool REL>
__device__ __forceinline__ void pass2_chunk(const float (&v)[32], fa_u32 (&pk)[16], fa_u64 cmul, fa_u64 negm,
                                            fa_u64& sum_a, fa_u64& sum_b) {
  pass2_part<REL, 0, 16>(v, pk, cmul, negm, sum_a, sum_b);
}

// State of one softmax warpgroup thread that a kv step reads and updates.
struct SoftmaxCtx {
  const FaParams& p;
  fa_u32 sb, t_s, t_o, t_p;
  int i, warp, qi, gb, gh;
  int half;  // decode variant: which 64 kv columns of a tile this thread owns (0 in the forward)
  float sc2;
  volatile int* abort_flag;
  float m_ref, l;
  fa_u32 cnt;
  const unsigned* rowbits;  // this query row of the mask bit matrix, or null
  ModLinear lin;            // a score_mod that is linear over kv
};

// One kv step of this warpgroup's tile.  The few tiles that need mask_mod or end beyond the
// sequence take one extra block after the scores are in registers.  VARIANT 2: one copy of the
// step, the block behind a run-time flag (head dim 64, where a second copy of the step costs more
// in the instruction cache than the branch: causal forward 100 against 108 us).  VARIANT 0 / 1: a
// copy without and a copy with the block (head dim 128, where the run-time flag made the common,
// unmasked steps 16 % slower).
template <int VARIANT>
__device__ __forceinline__ bool softmax_step(SoftmaxCtx& c, const int tile, const int mode, const bool masked_rt) {
  const bool masked = VARIANT == 2 ? masked_rt : VARIANT == 1;
  const FaParams& p = c.p;
  const fa_u32 sb = c.sb, t_o = c.t_o;
  const int i = c.i, qi = c.qi, gb = c.gb, gh = c.gh;
  const float sc2 = c.sc2;
  volatile int* abort_flag = c.abort_flag;
  float& m_ref = c.m_ref;
  float& l = c.l;
  fa_u32& cnt = c.cnt;
  const fa_u32 odd = ROT ? (cnt & 1u) : 0u;
  const fa_u32 t_s = c.t_s + odd * 64u, t_p = c.t_p + odd * 128u;
  // first key of this thread's columns (decode variant: the thread's 64-column half of the tile)
  const int n0 = tile * BN + (DECODE ? c.half * 64 : 0);
  const fa_u32 t_sh = DECODE ? t_s + c.half * 64 : t_s;
  constexpr bool REL = FA_HAS_SCORE_MOD;
  // What the scores are taken relative to (REL): the running maximum; 0 while the row has none, and where it is far below 0: a score_mod that
  // puts -1e30 in the place of scores makes it the maximum of a row whose first tile has no others, and added to that the
  // scores of later tiles are lost (at -1e4 all but their first bits).  From -64 on what they lose is below 2^-18.
  // A bias that is linear over the keys says by itself where the scores of the tile are: the bias of its first key takes the place of a
  // maximum that is more than 16 below, and of none.  (A large bias is then rounded once a tile: taken from 0 it would be rounded
  // at the eighth keys, at every key and in the sum again.)
  ModLinear lin = {};
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE) && defined(FA_SCORE_LINEAR_KV)
  lin = c.lin;
  const float bias0 = fa_score_add2(0.f, gb, gh, qi, n0);
  const float m_base = bias0 - m_ref <= 16.f ? m_ref : (fabsf(bias0) < -FA_NEG_INF ? bias0 : 0.f);
  lin.b = bias0 - m_base;
#else
  const float m_base = m_ref >= REL_FLOOR ? m_ref : 0.f;
#endif
  const bool use_mask = FA_HAS_MASK_MOD && mode == 1;
  const bool have_words = masked && use_mask && c.rowbits != nullptr;
  uint4 words = make_uint4(0u, 0u, 0u, 0u);
  // The mask words are on their way during the wait for the scores; not where few of many steps are partial (two tiles at head dim 64), where
  // they cost registers in every step
  constexpr bool LATE_WORDS = ROT && NQ == 2;
  if (!LATE_WORDS && have_words) words = mask_words<DECODE ? 2 : 4>(c.rowbits, n0);
  if (!fa_mbar_wait_warp(bar_addr(sb, BAR_S + i), cnt & 1u, abort_flag)) return false;
  fa_tc_fence_after();
  // ---- pass 1: the whole score row (128 fp32 values) comes into registers, chunk by chunk,
  // with the score_mod (when there is one) and the row maximum of a chunk computed
  // while the next chunk is on its way.  The S columns are free again as soon as the
  // last load has landed, long before the softmax of the step is done.
  float s0[32], s1[32], s2[32], s3[32];
  RowMax rm = {FA_NEG_INF, FA_NEG_INF, FA_NEG_INF, FA_NEG_INF};
  // (the host routes a non-positive scale, which would turn the maximum around, elsewhere)
#define FA_P1(V, C0)                                                                        \
  if (FA_HAS_SCORE_MOD || FA_ROUND_SCORES) mod_chunk<C0>(V, n0, qi, gb, gh, p.scale, sc2, -m_base, lin); \
  max_chunk(V, rm);
  fa_tmem_ld32(t_sh, s0);
  fa_tmem_wait_ld();
  fa_tmem_ld32(t_sh + 32, s1);
  FA_P1(s0, 0)
  fa_tmem_wait_ld();
  if (DECODE) {
    // two chunks are the whole share of this thread
    fa_tc_fence_before();
    fa_mbar_arrive(bar_addr(sb, BAR_SFREE2 + i));
    FA_P1(s1, 32)
  } else {
    fa_tmem_ld32(t_s + 64, s2);
    FA_P1(s1, 32)
    fa_tmem_wait_ld();
    fa_tmem_ld32(t_s + 96, s3);
    FA_P1(s2, 64)
    fa_tmem_wait_ld();
    if (EARLY_S) {
      fa_tc_fence_before();
      fa_mbar_arrive(bar_addr(sb, BAR_SFREE2 + i));
    }
    FA_P1(s3, 96)
  }
#undef FA_P1
  if (masked) {
    // (the row maximum taken on the way is of the unmasked scores: it is taken again)
    fa_u32 keep[DECODE ? 2 : 4];
    if (LATE_WORDS && have_words) words = mask_words<DECODE ? 2 : 4>(c.rowbits, n0);
    mask_bits(keep, use_mask, n0, qi, gb, gh, p.Skv, have_words, words);
    mask_apply(s0, keep[0]);
    mask_apply(s1, keep[1]);
    rm = {FA_NEG_INF, FA_NEG_INF, FA_NEG_INF, FA_NEG_INF};
    max_chunk(s0, rm);
    max_chunk(s1, rm);
    if (!DECODE) {
      mask_apply(s2, keep[DECODE ? 0 : 2]);
      mask_apply(s3, keep[DECODE ? 1 : 3]);
      max_chunk(s2, rm);
      max_chunk(s3, rm);
    }
  }
  float mx = fmaxf(fmaxf(rm.a, rm.b), fmaxf(rm.c, rm.d));
  if (!REL) mx *= sc2;
  // running maximum, raised lazily
  const float m_new = fmaxf(m_ref, REL ? m_base + mx : mx);
  bool need = false;
  float corr = 1.f;
  if (m_ref == FA_NEG_INF) {
    m_ref = m_new;  // nothing accumulated yet for this row
  } else if (m_new - m_ref > RESCALE_THRESHOLD) {
    need = true;
    corr = fa_ex2(m_ref - m_new);
    m_ref = m_new;
    l *= corr;
  }
  const float delta = REL && m_ref != FA_NEG_INF ? m_ref - m_base : 0.f;
  const bool rescale = cnt > 0 && __any_sync(0xffffffffu, need);
  if (cnt > 0 && (DECODE || rescale)) {
    // O is rescaled in place, and with separate P columns the previous PV product reads the P columns that are
    // about to be overwritten: it must be complete
    const fa_u32 last = cnt - 1;
    const int bar = ROT ? BAR_O + 2 * (int)(last & 1u) + i : BAR_O + i;
    if (!fa_mbar_wait_warp(bar_addr(sb, bar), (ROT ? last >> 1 : last) & 1u, abort_flag)) return false;
    fa_tc_fence_after();
  }
  if (rescale) {
#pragma unroll 1
    for (int c = 0; c < D / 16; ++c) {
      float o[16];
      fa_tmem_ld16(t_o + c * 16, o);
      fa_tmem_wait_ld();
#pragma unroll
      for (int e = 0; e < 16; ++e) o[e] *= corr;
      fa_tmem_st16f(t_o + c * 16, o);
    }
  }
  if (REL && __any_sync(0xffffffffu, delta != 0.f)) {
    // the maximum has moved (the first step of a row, hardly ever later) or is far below 0: the scores follow it
    const fa_u64 nd = fa_f2(-delta, -delta);
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
      fa_f2_unpack(fa_add2(fa_f2(s0[e], s0[e + 1]), nd), s0[e], s0[e + 1]);
      fa_f2_unpack(fa_add2(fa_f2(s1[e], s1[e + 1]), nd), s1[e], s1[e + 1]);
      if (!DECODE) {
        fa_f2_unpack(fa_add2(fa_f2(s2[e], s2[e + 1]), nd), s2[e], s2[e + 1]);
        fa_f2_unpack(fa_add2(fa_f2(s3[e], s3[e + 1]), nd), s3[e], s3[e + 1]);
      }
    }
  }
  // ---- pass 2: p = 2^(x * scale - m) and the row sum; P goes to TMEM as 16-bit pairs.
  // (Packed 16-bit exponentials - ex2.approx.f16x2, one SFU operation per pair - were measured
  // slower: 143 against 131 us, the conversions around them cost more than the SFU time they save.)
  const float m_use = (m_ref == FA_NEG_INF) ? 0.f : m_ref;
  const fa_u64 negm = fa_f2(-m_use, -m_use);
  const fa_u64 cmul = fa_f2(sc2, sc2);
  fa_u64 sum_a = fa_f2(0.f, 0.f), sum_b = fa_f2(0.f, 0.f);
  {
    fa_u32 pk[16];
    const fa_u32 t_ph = DECODE ? t_p + c.half * 32 : t_p;  // (the other 32 columns of the lane stay zero)
    pass2_chunk<REL>(s0, pk, cmul, negm, sum_a, sum_b);
    fa_tmem_st16(t_ph, pk);
    pass2_chunk<REL>(s1, pk, cmul, negm, sum_a, sum_b);
    fa_tmem_st16(t_ph + 16, pk);
    if (!DECODE) {
      pass2_chunk<REL>(s2, pk, cmul, negm, sum_a, sum_b);
      fa_tmem_st16(t_p + 32, pk);
      if (SPLIT_P) {
        pass2_part<REL, 0, 8>(s3, pk, cmul, negm, sum_a, sum_b);
        fa_tmem_wait_st();
        fa_tc_fence_before();
        fa_mbar_arrive(bar_addr(sb, BAR_P + i));
        pass2_part<REL, 8, 16>(s3, pk, cmul, negm, sum_a, sum_b);
      } else {
        pass2_chunk<REL>(s3, pk, cmul, negm, sum_a, sum_b);
      }
      fa_tmem_st16(t_p + 48, pk);
    }
  }
  float sum;
  {
    float a0, a1;
    fa_f2_unpack(fa_add2(sum_a, sum_b), a0, a1);
    sum = a0 + a1;
  }
  l += sum;
  fa_tmem_wait_st();
  fa_tc_fence_before();
  fa_mbar_arrive(bar_addr(sb, (SPLIT_P ? BAR_P2 : BAR_P + 2 * (int)odd) + i));
  ++cnt;
  return true;
}

#if FA_DTYPE == FA_DT_F32
// One kv step of a tile with fp32 inputs.  The scores are gone through twice, 32 columns at a time, so that the
// output row (acc, 64 values) fits into the registers beside them: first for the row maximum, then
// for the exponentials and their parts.  A score_mod that adds something is evaluated in the first
// pass only and its results are written back; one that only multiplies is cheap enough for both.
#if FA_HAS_SCORE_MOD && !defined(FA_SCORE_MUL_ONLY)
constexpr bool WRITE_BACK = true;
#else
constexpr bool WRITE_BACK = false;
#endif
// the scores of 32 columns in log2 units (raw without a score_mod: the exponent's FMA applies the scale then)
template <int C0>
__device__ __forceinline__ void mod32_f32(float (&v)[32], const SoftmaxCtx& c, int n0) {
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_MUL_ONLY)
#pragma unroll
  for (int e = 0; e < 32; ++e) v[e] *= fa_score_mul(0.f, c.gb, c.gh, c.qi, n0 | (C0 + e)) * c.sc2;
#elif FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE)
  // (an additive bias is applied before the change to log2 units, as in fa_fwd.cuh: folding the factor into it would round
  //  a large bias at another place.  The FMA is written out: which product of  score * scale + a * b  is fused is otherwise
  //  up to the compiler, and the backward has to see the same scores: with ALiBi, S856, gradients were off by 1.0e-5 to 1.3e-5
  //  instead of 0.8e-5 to 1.1e-5 where the two differed)
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    const int kv = n0 | (C0 + e);
    v[e] = fmaf(v[e], fa_score_mul(0.f, c.gb, c.gh, c.qi, kv) * c.p.scale, fa_score_add(0.f, c.gb, c.gh, c.qi, kv)) * FA_LOG2E;
  }
#elif FA_HAS_SCORE_MOD
#pragma unroll
  for (int e = 0; e < 32; ++e) v[e] = fa_score_mod(v[e] * c.p.scale, c.gb, c.gh, c.qi, n0 | (C0 + e)) * FA_LOG2E;
#endif
}
__device__ __forceinline__ bool softmax_step_f32(SoftmaxCtx& c, float (&acc)[D], const int tile, const int mode, const bool masked) {
  const FaParams& p = c.p;
  const fa_u32 t_s = c.t_s;
  const int n0 = tile * BN;
  if (!fa_mbar_wait_warp(bar_addr(c.sb, BAR_S + c.i), c.cnt & 1u, c.abort_flag)) return false;
  fa_tc_fence_after();
  float a[32], b[32];
  constexpr bool mod = FA_HAS_SCORE_MOD;
  fa_u32 keep[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
  fa_tmem_ld32(t_s, a);
  if (masked) {
    const bool have_words = FA_HAS_MASK_MOD && mode == 1 && c.rowbits != nullptr;
    uint4 words = make_uint4(0u, 0u, 0u, 0u);
    if (have_words) words = mask_words<4>(c.rowbits, n0);
    mask_bits(keep, FA_HAS_MASK_MOD && mode == 1, n0, c.qi, c.gb, c.gh, p.Skv, have_words, words);
  }
  float mx0 = FA_NEG_INF, mx1 = FA_NEG_INF;
#define FA_P1(V, N, C)                                                                                  \
  fa_tmem_wait_ld();                                                                                    \
  if ((C) + 32 < BN) fa_tmem_ld32(t_s + (C) + 32, N);                                                   \
  mod32_f32<C>(V, c, n0);                                                                               \
  if (masked) mask_apply(V, keep[(C) >> 5]);                                                            \
  if (WRITE_BACK || masked) fa_tmem_st32(t_s + (C), V);                                                 \
  _Pragma("unroll") for (int e = 0; e < 32; e += 4) {                                                   \
    mx0 = fa_max3(mx0, V[e], V[e + 1]);                                                                 \
    mx1 = fa_max3(mx1, V[e + 2], V[e + 3]);                                                             \
  }
  FA_P1(a, b, 0) FA_P1(b, a, 32) FA_P1(a, b, 64) FA_P1(b, a, 96)
#undef FA_P1
  if (c.cnt > 0) fa_tmem_ld32(c.t_o, a);
  float mx = fmaxf(mx0, mx1);
  if (!mod) mx *= c.sc2;
  const float m_new = fmaxf(c.m_ref, mx);
  float corr = 1.f;
  if (c.m_ref == FA_NEG_INF) {
    c.m_ref = m_new;
  } else if (m_new - c.m_ref > RESCALE_THRESHOLD) {
    corr = fa_ex2(c.m_ref - m_new);
    c.m_ref = m_new;
    c.l *= corr;
  }
  if (c.cnt > 0) {
    // S of this step was issued behind P.V of the last one, so that product is complete too
    fa_tmem_wait_ld();
    fa_tmem_ld32(c.t_o + 32, b);
#pragma unroll
    for (int e = 0; e < 32; ++e) acc[e] = (acc[e] + a[e]) * corr;
    fa_tmem_wait_ld();
#pragma unroll
    for (int e = 0; e < 32; ++e) acc[32 + e] = (acc[32 + e] + b[e]) * corr;
  }
  if (WRITE_BACK || masked) fa_tmem_wait_st();
  fa_tmem_ld32(t_s, a);
  const float m_use = (c.m_ref == FA_NEG_INF) ? 0.f : c.m_ref;
  const fa_u64 negm = fa_f2(-m_use, -m_use);
  const float cm = mod ? 1.f : c.sc2;
  const fa_u64 cmul = fa_f2(cm, cm);
  fa_u64 sum_a = fa_f2(0.f, 0.f), sum_b = fa_f2(0.f, 0.f);
#define FA_P2(V, N, C)                                                                                  \
  fa_tmem_wait_ld();                                                                                    \
  if ((C) + 32 < BN) fa_tmem_ld32(t_s + (C) + 32, N);                                                   \
  if (mod && !WRITE_BACK && !masked) mod32_f32<C>(V, c, n0);                                            \
  _Pragma("unroll") for (int hf = 0; hf < 2; ++hf) {                                                    \
    fa_u32 hi[8], mid[8], lo[8];                                                                        \
    _Pragma("unroll") for (int e = 0; e < 8; ++e) {                                                     \
      float x0, x1;                                                                                     \
      fa_f2_unpack(fa_fma2(fa_f2(V[16 * hf + 2 * e], V[16 * hf + 2 * e + 1]), cmul, negm), x0, x1);     \
      const fa_u64 pf = fa_f2(fa_ex2(x0), fa_ex2(x1));                                                  \
      if (e & 1) sum_b = fa_add2(sum_b, pf);                                                            \
      else sum_a = fa_add2(sum_a, pf);                                                                  \
      fa_split3(pf, hi[e], mid[e], lo[e]);                                                              \
    }                                                                                                   \
    fa_tmem_st8(t_s + (C) + 8 * hf, hi);                                                                \
    fa_tmem_st8(t_s + (C) + 16 + 8 * hf, mid);                                                          \
    fa_tmem_st8(t_s + 128 + (C) / 2 + 8 * hf, lo);                                                      \
  }
  FA_P2(a, b, 0) FA_P2(b, a, 32) FA_P2(a, b, 64) FA_P2(b, a, 96)
#undef FA_P2
  float s0, s1;
  fa_f2_unpack(fa_add2(sum_a, sum_b), s0, s1);
  c.l += s0 + s1;
  fa_tmem_wait_st();
  fa_tc_fence_before();
  fa_mbar_arrive(bar_addr(c.sb, BAR_P + c.i));
  ++c.cnt;
  return true;
}
#endif

}  // namespace fa_tc

extern "C" __global__ void __launch_bounds__(fa_tc::NT, fa_tc::NQ == 1 ? 2 : 1) fa_fwd_tc_kernel(const __grid_constant__ FaTcParams P) {
  using namespace fa_tc;
  const FaParams& p = P.p;
  extern __shared__ unsigned char smem_raw[];
  // a launch that does not fit the shared-memory map below (a host library built for another
  // version of this file) is refused before anything is written
  if (fa_dynamic_smem_size() < (fa_u32)SMEM_BYTES || blockDim.x != NT) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicOr(p.status, FA_STATUS_BAD_LAUNCH);
    return;
  }
  FA_MOD_BUFS_INIT(p);
  fa_grid_wait();
  const fa_u32 raw = fa_smem_u32(smem_raw);
  const fa_u32 sb = (raw + 1023u) & ~1023u;  // shared-window address of the aligned base
  unsigned char* sm = smem_raw + (sb - raw);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#if FA_TC_DECODE
  const int split = blockIdx.x, h = blockIdx.y, b = blockIdx.z;  // grid: (kv shares, heads, batch)
  const int m0 = 0;
#else
  const int pair = gridDim.z - 1 - blockIdx.z;  // grid: (heads, batch, tile pairs), the last pair first
  const int h = blockIdx.x, b = blockIdx.y;
  const int m0 = pair * NQ * BM;
#endif
  const int hk = h / (p.Hq / p.Hkv);
  const int gb = b + p.b_off, gh = h + p.h_off;

  volatile int* misc = (volatile int*)(sm + OFF_MISC);  // [0] tmem base, [1] abort, [2] nsteps
  volatile fa_u32* sched = (volatile fa_u32*)(sm + OFF_SCHED);
  unsigned char* cls = sm + OFF_CLS;

  // The BlockMask table reads of this CTA go out first: the two counts and, speculatively, this
  // thread's entry of the two index lists, for both query tiles.  They are all issued before any is
  // used (one round trip to memory instead of a chain of four dependent ones) and they are in flight
  // while the barriers are set up and TMEM is allocated.
  constexpr int NI = DECODE ? 1 : NQ;
  const int ntiles = min((p.Skv + BN - 1) / BN, MAXT);
  const bool tables = p.t.kv_num != nullptr;
  const int tpb = tables ? (p.t.nKV == 1 ? ntiles : p.t.KVB / BN) : 1;
  const int bi0 = tid / tpb, ti0 = tid - bi0 * tpb;
  long long rows[NI];
  int num[NI][2], blk[NI][2];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int mi = m0 + i * BM;
    const int bm = p.t.mB == 1 ? 0 : b, hm = p.t.mH == 1 ? 0 : h;
    const int qblk = tables ? min(mi / p.t.QB, p.t.nQ - 1) : 0;
    rows[i] = ((long long)bm * p.t.mH + hm) * p.t.nQ + qblk;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const int* nump = which ? p.t.full_kv_num : p.t.kv_num;
      const int* idxp = which ? p.t.full_kv_idx : p.t.kv_idx;
      const bool have = tables && nump != nullptr && mi < p.Sq;
      num[i][which] = have ? nump[rows[i]] : 0;
      blk[i][which] = (have && bi0 < p.t.nKV) ? idxp[rows[i] * p.t.nKV + bi0] : 0;
    }
  }

  // ---- set-up: barriers, TMEM, kv schedule ---------------------------------------------
  if (tid == 0) {
    fa_mbar_init(bar_addr(sb, BAR_Q), 1);
    for (int s = 0; s < NSTAGE; ++s) {
      fa_mbar_init(bar_addr(sb, BAR_KFULL + s), 1);
      fa_mbar_init(bar_addr(sb, BAR_KEMPTY + s), ROT ? NQ : 1);
      fa_mbar_init(bar_addr(sb, BAR_VFULL + s), 1);
      fa_mbar_init(bar_addr(sb, BAR_VEMPTY + s), ROT ? NQ : 1);
    }
    for (int i = 0; i < 2; ++i) {
      fa_mbar_init(bar_addr(sb, BAR_S + i), 1);
      fa_mbar_init(bar_addr(sb, BAR_P + i), 128);
      fa_mbar_init(bar_addr(sb, BAR_P + 2 + i), 128);
      fa_mbar_init(bar_addr(sb, BAR_O + i), 1);
      fa_mbar_init(bar_addr(sb, BAR_O + 2 + i), 1);
      fa_mbar_init(bar_addr(sb, BAR_SFREE2 + i), 128);
    }
    fa_mbar_init(bar_addr(sb, BAR_LAG), 1);
    fa_mbar_init_fence();
    misc[1] = 0;
    misc[2] = 0;
    // the query tiles do not depend on the kv schedule: their loads start now and run while the
    // schedule is being built
    fa_tma_prefetch_desc(&P.tq);
    // (decode variant: the query map's box is 64 rows and each warpgroup's tile gets the queries
    //  twice, in rows 0-63 and in rows 64-127; rows beyond Sq are out of range and read as zero)
    fa_mbar_expect_tx(bar_addr(sb, BAR_Q), Q_BYTES);
    for (int i = 0; i < NQ; ++i)
      for (int a = 0; a < ATOMS; ++a) {
        if (DECODE) {
          fa_tma_load_4d(sb + (i * ATOMS + a) * ATOM_BYTES, &P.tq, bar_addr(sb, BAR_Q), a * 64, 0, h, b);
          fa_tma_load_4d(sb + (i * ATOMS + a) * ATOM_BYTES + 64 * 128, &P.tq, bar_addr(sb, BAR_Q), a * 64, 0, h, b);
        } else {
          fa_tma_load_4d(sb + (i * ATOMS + a) * ATOM_BYTES, &P.tq, bar_addr(sb, BAR_Q), a * 64, m0 + i * BM, h, b);
        }
      }
  }
  for (int i = tid; i < 2 * MAXT; i += NT) cls[i] = 0;
  if (warp == WARP_MMA) fa_tmem_alloc(sb + OFF_MISC, TMEM_COLS);
  __syncthreads();
  // class of every kv tile for both query tiles: 0 skip, 1 apply mask_mod, 2 full (from the table
  // entries read at the top of the kernel)
  {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int mi = m0 + i * BM;
      if (mi >= p.Sq) continue;
      if (!tables) {
        for (int t = tid; t < ntiles; t += NT) cls[i * MAXT + t] = FA_HAS_MASK_MOD ? 1 : 2;
        continue;
      }
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const int* idxp = which ? p.t.full_kv_idx : p.t.kv_idx;
        const int n = min(max(num[i][which], 0), p.t.nKV) * tpb;
        if (tid < n) {
          const int t = min(max(blk[i][which], 0), p.t.nKV - 1) * tpb + ti0;
          if (t < ntiles) cls[i * MAXT + t] = (unsigned char)(which ? 2 : 1);
        }
        for (int e = tid + NT; e < n; e += NT) {  // (more list entries than threads)
          const int bi = e / tpb, ti = e - bi * tpb;
          const int t = min(max(idxp[rows[i] * p.t.nKV + bi], 0), p.t.nKV - 1) * tpb + ti;
          if (t < ntiles) cls[i * MAXT + t] = (unsigned char)(which ? 2 : 1);
        }
      }
    }
  }
  __syncthreads();
  // The kv schedule: the listed tiles in ascending order, compacted by the first 256 threads (one
  // tile each) with a ballot per warp and a prefix over the eight warp counts.
  {
    int* wcount = (int*)(sm + OFF_WCNT);
    const bool mine = tid < MAXT;
    const unsigned char c0 = (mine && tid < ntiles) ? cls[tid] : 0;
    const unsigned char c1 = (!DECODE && NQ == 2 && mine && tid < ntiles) ? cls[MAXT + tid] : 0;
    const bool listed = (c0 | c1) != 0;
    const unsigned vote = __ballot_sync(0xffffffffu, listed);
    if (mine && lane == 0) wcount[warp] = __popc(vote);
    __syncthreads();
    if (mine) {
      int before = 0, total = 0;
      for (int w = 0; w < MAXT / 32; ++w) {
        const int n = wcount[w];
        before += w < warp ? n : 0;
        total += n;
      }
      const int pos = before + __popc(vote & ((1u << lane) - 1u));
#if FA_TC_DECODE
      // this CTA's share of the listed kv tiles; entry k of the share belongs to warpgroup k % 2
      const int per = (total + (int)gridDim.x - 1) / (int)gridDim.x;
      const int lo = split * per, hi = min(total, lo + per);
      if (listed && pos >= lo && pos < hi) {
        sched[pos - lo] = (fa_u32)tid | ((fa_u32)c0 << 16);
      }
      if (tid == 0) {
        const int k = max(hi - lo, 0);
        sched[k] = 0;  // an odd share leaves the second warpgroup without a tile in the last step
        misc[2] = (k + 1) / 2;
        misc[3] = k;
      }
#else
      if (listed) {
        sched[pos] = (fa_u32)tid | ((fa_u32)c0 << 16) | ((fa_u32)c1 << 24);
      }
      if (tid == 0) {
        misc[2] = total;
        misc[3] = total;
      }
#endif
    }
  }
  fa_tc_fence_before();
  __syncthreads();
  fa_tc_fence_after();
  const fa_u32 tmem = (fa_u32)misc[0];
  const int nsteps = misc[2];   // steps of the softmax / MMA loops
  const int nloads = misc[3];   // kv tiles the producer brings in (two per step in the decode variant)
  volatile int* abort_flag = misc + 1;

  if (warp >= NSOFT) fa_setmaxnreg_dec<REGS_OTHER>();
  if (warp == WARP_PRODUCER) {
    // ================================ TMA producer =======================================
    if (lane == 0) {
      fa_tma_prefetch_desc(&P.tk);
      fa_tma_prefetch_desc(&P.tv);
      // a CTA without kv tiles still has to see its query loads land before it may exit
      bool ok = nloads > 0 || fa_mbar_wait(bar_addr(sb, BAR_Q), 0, abort_flag);
      for (int j = 0; j < nloads && ok; ++j) {
        const int s = j % NSTAGE;
        const fa_u32 ph = (fa_u32)((j / NSTAGE) & 1);
        const int n0 = (int)(sched[j] & 0xffffu) * BN;
        if (j >= NSTAGE) ok = fa_mbar_wait(bar_addr(sb, BAR_KEMPTY + s), ph ^ 1u, abort_flag);
        if (!ok) break;
        fa_mbar_expect_tx(bar_addr(sb, BAR_KFULL + s), KV_STAGE);
        for (int a = 0; a < ATOMS; ++a)
          fa_tma_load_4d(sb + OFF_K + s * KV_STAGE + a * ATOM_BYTES, &P.tk, bar_addr(sb, BAR_KFULL + s), a * 64, n0, hk, b);
        if (j >= NSTAGE) ok = fa_mbar_wait(bar_addr(sb, BAR_VEMPTY + s), ph ^ 1u, abort_flag);
        if (!ok) break;
        fa_mbar_expect_tx(bar_addr(sb, BAR_VFULL + s), KV_STAGE);
        for (int a = 0; a < ATOMS; ++a)
          fa_tma_load_4d(sb + OFF_V + s * KV_STAGE + a * ATOM_BYTES, &P.tv, bar_addr(sb, BAR_VFULL + s), a * 64, n0, hk, b);
      }
    }
  } else if (DECODE && (warp == WARP_MMA || warp == WARP_MMA_B)) {
    // ============ decode variant: warp A issues the S products, warp B the PV products ======
    // With P in its own TMEM columns the two streams only meet through the softmax warps, so each
    // issuer waits on its own barriers and the waits of one overlap the issue of the other.
    if (lane == 0 && nsteps > 0) {
      constexpr fa_u32 HI = fa_desc_hi_sw128();
      if (warp == WARP_MMA) {
        constexpr fa_u32 IDESC_S = fa_idesc(DT, BM, BN, 0, 0);
        bool ok = fa_mbar_wait(bar_addr(sb, BAR_Q), 0, abort_flag);
        fa_u32 nsi[2] = {0, 0};
        for (int j = 0; j < nsteps && ok; ++j) {
          // (the warpgroups take the CTA's share of the kv tiles in turn)
          for (int i = 0; i < NQ && ok; ++i) {
            const int t = 2 * j + i, s = t % NSTAGE;
            if (!(sched[t] >> 16)) continue;
            ok = fa_mbar_wait(bar_addr(sb, BAR_KFULL + s), (fa_u32)((t / NSTAGE) & 1), abort_flag);
            if (!ok) break;
            if (nsi[i] > 0) {
              ok = fa_mbar_wait(bar_addr(sb, BAR_SFREE2 + i), (nsi[i] - 1) & 1u, abort_flag);
              if (!ok) break;
            }
            fa_tc_fence_after();
            const fa_u32 loQ = fa_desc_lo(sb + i * ATOMS * ATOM_BYTES, 16), loK = fa_desc_lo(sb + OFF_K + s * KV_STAGE, 16);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              const fa_u32 koff = ((kk / 4) * ATOM_BYTES + (kk % 4) * 32) >> 4;
              fa_mma_ss(tmem + COL_S + i * BN, fa_desc_make(loQ + koff, HI), fa_desc_make(loK + koff, HI), IDESC_S, kk > 0);
            }
            fa_mma_commit(bar_addr(sb, BAR_S + i));
            fa_mma_commit(bar_addr(sb, BAR_KEMPTY + s));
            ++nsi[i];
          }
        }
      } else {
        constexpr fa_u32 IDESC_O = fa_idesc(DT, BM, D, 0, 1);
        bool ok = true;
        fa_u32 cnt[2] = {0, 0};
        for (int j = 0; j < nsteps && ok; ++j) {
          for (int i = 0; i < NQ && ok; ++i) {
            const int t = 2 * j + i, s = t % NSTAGE;
            if (!(sched[t] >> 16)) continue;
            ok = fa_mbar_wait(bar_addr(sb, BAR_VFULL + s), (fa_u32)((t / NSTAGE) & 1), abort_flag);
            if (!ok) break;
            ok = fa_mbar_wait(bar_addr(sb, BAR_P + i), cnt[i] & 1u, abort_flag);
            if (!ok) break;
            fa_tc_fence_after();
            const fa_u32 loV = fa_desc_lo(sb + OFF_V + s * KV_STAGE, ATOM_BYTES);
            const fa_u32 acc = cnt[i] > 0;
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk)
              fa_mma_ts(tmem + COL_O + i * D, tmem + COL_P + i * 64 + kk * 8, fa_desc_make(loV + kk * 128, HI), IDESC_O, acc | (kk > 0));
            fa_mma_commit(bar_addr(sb, BAR_O + i));
            fa_mma_commit(bar_addr(sb, BAR_VEMPTY + s));
            ++cnt[i];
          }
        }
      }
    }
  } else if (ROT && warp >= WARP_MMA && warp < WARP_MMA + NQ) {
    // ============ head dim 64: an issuing warp per query tile ==============================
    // S(j+1) lies over the P columns of step j-1, whose product this warp has issued before it.  The whole warp runs the loop and one elected lane issues: in uniform control flow the
    // operands of tcgen05.mma sit in uniform registers, which makes the instructions cheaper to issue than from a
    // single-lane branch.  (With one warp for both tiles the issue of one tile's products delayed the other's.)
    const int i = __shfl_sync(0xffffffffu, warp - WARP_MMA, 0);
    const bool leader = fa_elect_one();
    const fa_u32 tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    const int nsteps_u = __shfl_sync(0xffffffffu, nsteps, 0);
    constexpr fa_u32 IDESC_S = fa_idesc(DT, BM, BN, 0, 0);
    constexpr fa_u32 IDESC_O = fa_idesc(DT, BM, D, 0, 1);
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    bool ok = nsteps_u == 0 || fa_mbar_wait_all(bar_addr(sb, BAR_Q), 0, abort_flag);
    fa_u32 ns = 0, cnt = 0;  // S and PV products issued so far
    auto word = [&](int j) { return __shfl_sync(0xffffffffu, sched[j], 0); };
    auto active = [&](fa_u32 w) { return ((w >> (16 + 8 * i)) & 0xffu) != 0u; };
    auto wait_k = [&](int j) { return fa_mbar_wait_all(bar_addr(sb, BAR_KFULL + j % NSTAGE), (fa_u32)((j / NSTAGE) & 1), abort_flag); };
    const fa_u32 loQ = fa_desc_lo(sb + i * ATOMS * ATOM_BYTES, 16);
    // S(j), and K of the step is released (every step's K is waited for before that, with or without a product)
    auto do_s = [&](int j, fa_u32 wj) {
      if (active(wj)) {
        if (ns > 0 && !fa_mbar_wait_all(bar_addr(sb, BAR_SFREE2 + i), (ns - 1) & 1u, abort_flag)) return false;
        fa_tc_fence_after();
        const fa_u32 loK = fa_desc_lo(sb + OFF_K + (j % NSTAGE) * KV_STAGE, 16);
        const fa_u32 t_s = tmem_u + COL_S + i * S_STRIDE + (ns & 1u) * 64u;
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            fa_mma_ss(t_s, fa_desc_make(loQ + kk * 2, HI), fa_desc_make(loK + kk * 2, HI), IDESC_S, kk > 0);
          fa_mma_commit(bar_addr(sb, BAR_S + i));
        }
        ++ns;
      }
      if (leader) fa_mma_commit(bar_addr(sb, BAR_KEMPTY + j % NSTAGE));
      return true;
    };
    fa_u32 w = word(0);
    if (ok && nsteps_u > 0) {
      ok = wait_k(0);
      // The first tile starts when the first PV product of the second is complete, and the two stay apart like that: in step, the loads
      // and waits of one do not run under the exponentials of the other.  us, in step / apart by the loads / by this: dense B2 H8 S8192 420 / 375 /
      // 380, B1 H4 S8192 113.5 / 112.6 / 109.5, S2304 (16 heads) 37.7 / 37.4 / 35.0, causal B1 H8 S8192 109 / 111 / 103, B2 H8 S8192 206 / 195 / 191,
      // S4096 61.9 / 60.2 / 58.8, B8 H8 S4096 226 / 212 / 214, ALiBi B2 H8 S8192 493 / 445 / 442.  The second tile goes first since under a
      // causal mask it has a step more, and without one it is faster too (first tile first, by the loads: causal B2 H8 S8192 199, B1 H8
      // 110, dense B1 H8 S8192 205 against 200).  Turns at every step, each tile's scores behind the other's loads, were slower (dense B2 H8 S8192 415).
      if (NQ == 2 && i == 0 && nsteps_u > 1 && ((w >> 24) & 0xffu) != 0u && ((word(1) >> 24) & 0xffu) != 0u && active(w))
        ok = ok && fa_mbar_wait_all(bar_addr(sb, BAR_LAG), 0, abort_flag);
      ok = ok && do_s(0, w);
    }
    for (int j = 0; j < nsteps_u && ok; ++j) {
      const bool more = j + 1 < nsteps_u;
      const fa_u32 w1 = more ? word(j + 1) : 0u;
      // S(j+1) as soon as the scores of step j are in registers, PV(j) when P is there
      if (more) ok = wait_k(j + 1) && do_s(j + 1, w1);
      if (ok) ok = fa_mbar_wait_all(bar_addr(sb, BAR_VFULL + j % NSTAGE), (fa_u32)((j / NSTAGE) & 1), abort_flag);
      if (!ok) break;
      if (active(w)) {
        const fa_u32 loV = fa_desc_lo(sb + OFF_V + (j % NSTAGE) * KV_STAGE, ATOM_BYTES);
        const fa_u32 t_p = tmem_u + COL_S + i * S_STRIDE + (cnt & 1u) * 128u, t_o = tmem_u + COL_O + i * D;
        const int odd = 2 * (int)(cnt & 1u) + i;
        ok = fa_mbar_wait_all(bar_addr(sb, BAR_P + odd), (cnt >> 1) & 1u, abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < BN / 16; ++kk)
            fa_mma_ts(t_o, t_p + kk * 8, fa_desc_make(loV + kk * 128, HI), IDESC_O, (cnt > 0) | (kk > 0));
          fa_mma_commit(bar_addr(sb, BAR_O + odd));
          if (NQ == 2 && i == 1 && cnt == 0) fa_mma_commit(bar_addr(sb, BAR_LAG));
        }
        ++cnt;
      }
      if (leader) fa_mma_commit(bar_addr(sb, BAR_VEMPTY + j % NSTAGE));
      w = w1;
    }
  } else if (!DECODE && !ROT && warp == WARP_MMA) {
    // ============ one MMA issuer for both query tiles ======================================
    // The whole warp runs the loop and one elected lane issues: in uniform control flow the operands of tcgen05.mma
    // sit in uniform registers, which makes the instructions cheaper to issue than from a single-lane branch.
    // Everything a product needs besides what the softmax hands over (the K / V tile, the modes of the step) is
    // waited for before that, so that the products follow the hand-over at once.
    const bool leader = fa_elect_one();
    const fa_u32 tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    const int nsteps_u = __shfl_sync(0xffffffffu, nsteps, 0);
    constexpr fa_u32 IDESC_S = fa_idesc(DT, BM, BN, 0, 0);
    constexpr fa_u32 IDESC_O = fa_idesc(DT, BM, D, 0, 1);
    bool ok = nsteps_u == 0 || fa_mbar_wait_all(bar_addr(sb, BAR_Q), 0, abort_flag);
    fa_u32 cnt[2] = {0, 0};  // PV products of each tile issued so far
    // Descriptors: constant high word; the low word (start address and MN-chunk distance in
    // 16-byte units) is stepped with one add per k-step.
    constexpr fa_u32 HI = fa_desc_hi_sw128();
    auto word = [&](int j) { return __shfl_sync(0xffffffffu, sched[j], 0); };
    auto active = [&](fa_u32 w, int i) { return ((w >> (16 + 8 * i)) & 0xffu) != 0u; };
    auto wait_k = [&](int j) { return fa_mbar_wait_all(bar_addr(sb, BAR_KFULL + j % NSTAGE), (fa_u32)((j / NSTAGE) & 1), abort_flag); };
    auto have_k = [&](int j) { return __all_sync(0xffffffffu, fa_mbar_try(bar_addr(sb, BAR_KFULL + j % NSTAGE), (fa_u32)((j / NSTAGE) & 1))) != 0; };
    auto wait_v = [&](int j) { return fa_mbar_wait_all(bar_addr(sb, BAR_VFULL + j % NSTAGE), (fa_u32)((j / NSTAGE) & 1), abort_flag); };
    // S_i = Q_i K^T for step j
    auto issue_s = [&](int j, int i) {
      const int s = j % NSTAGE;
      const fa_u32 loQ = fa_desc_lo(sb + i * ATOMS * ATOM_BYTES, 16);
      const fa_u32 loK = fa_desc_lo(sb + OFF_K + s * KV_STAGE, 16);
      if (leader) {
#pragma unroll
        for (int pr = 0; pr < NPROD; ++pr) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const fa_u32 koff = ((kk / 4) * ATOM_BYTES + (kk % 4) * 32) >> 4;
            const fa_u32 pa = (PROD_A[pr] * ATOM_BYTES) >> 4, pb = (PROD_B[pr] * ATOM_BYTES) >> 4;
            fa_mma_ss(tmem_u + COL_S + i * S_STRIDE, fa_desc_make(loQ + pa + koff, HI), fa_desc_make(loK + pb + koff, HI), IDESC_S, pr > 0 || kk > 0);
          }
        }
        fa_mma_commit(bar_addr(sb, BAR_S + i));
      }
    };
    // O_i += P_i V for step j (P_i: 16-bit, from the first column of S_i on; fp32: three parts, and O_i = P_i V)
    auto issue_pv = [&](int j, int i) {
      const int s = j % NSTAGE;
      const fa_u32 loV = fa_desc_lo(sb + OFF_V + s * KV_STAGE, ATOM_BYTES);
      const fa_u32 acc = !F32 && cnt[i] > 0;
      const fa_u32 t_p = tmem_u + COL_S + i * S_STRIDE, t_o = tmem_u + COL_O + i * D;
      constexpr int K1 = SPLIT_P ? 6 : BN / 16;
      if (leader) {
#pragma unroll
        for (int pr = 0; pr < NPROD; ++pr) {
#pragma unroll
          for (int kk = 0; kk < K1; ++kk)
            fa_mma_ts(t_o, t_p + (!F32 ? kk * 8 : (PROD_A[pr] == 2 ? 128 + kk * 8 : (kk >> 1) * 32 + PROD_A[pr] * 16 + (kk & 1) * 8)),
                      fa_desc_make(loV + ((PROD_B[pr] * ATOM_BYTES) >> 4) + kk * 128, HI), IDESC_O, acc | (pr > 0 || kk > 0));
        }
      }
      if (SPLIT_P) {
        if (!fa_mbar_wait_all(bar_addr(sb, BAR_P2 + i), cnt[i] & 1u, abort_flag)) return false;
        fa_tc_fence_after();
      }
      if (leader) {
#pragma unroll
        for (int kk = K1; kk < BN / 16; ++kk)
          fa_mma_ts(t_o, t_p + kk * 8, fa_desc_make(loV + kk * 128, HI), IDESC_O, 1u);
        fa_mma_commit(bar_addr(sb, BAR_O + i));
      }
      ++cnt[i];
      return true;
    };
    fa_u32 w = word(0);
    if (ok && nsteps_u > 0) {
      ok = wait_k(0);
      if (ok) {
        fa_tc_fence_after();
        for (int i = 0; i < NQ; ++i)
          if (active(w, i)) issue_s(0, i);
        if (leader) fa_mma_commit(bar_addr(sb, BAR_KEMPTY + 0));
      }
    }
    {
      // P overwrites the S columns here (D = 128, fp32), so the products of one tile form a chain  PV_i(j), S_i(j+1),
      // PV_i(j+1) ...  One warp issues the two chains in turn, PV_0(j) S_0(j+1) PV_1(j) S_1(j+1), so that the
      // products of a tile run as one block while the other tile is in its softmax.  (With an issuing warp
      // per tile the tensor core took instructions of both in turn, both tiles got their scores at the
      // same time, and the products of one never ran under the softmax of the other: clock stamps of a
      // step showed both waiting for the tensor core and both in the softmax together.)
      for (int j = 0; j < nsteps_u && ok; ++j) {
        const bool more = j + 1 < nsteps_u;
        const fa_u32 w_next = more ? word(j + 1) : 0u;
        // (every step waits for its stage to be full before it releases it, with or without a product; where K of the
        // next step is still on its way, PV of the first tile goes first)
        ok = wait_v(j);
        bool k_there = !more || (NSTAGE > 1 && have_k(j + 1));
#pragma unroll (F32 ? 1 : NQ)
        for (int i = 0; i < NQ; ++i) {
          if (!ok) break;
          if (active(w, i)) {
            ok = fa_mbar_wait_all(bar_addr(sb, BAR_P + i), cnt[i] & 1u, abort_flag);
            if (!ok) break;
            fa_tc_fence_after();
            ok = issue_pv(j, i);
            if (!ok) break;
          }
          if (i == NQ - 1 && leader) fa_mma_commit(bar_addr(sb, BAR_VEMPTY + j % NSTAGE));
          if (!k_there) {
            ok = wait_k(j + 1);
            if (!ok) break;
            k_there = true;
            fa_tc_fence_after();
          }
          // S of the next step overwrites the columns P was read from: it follows the PV product
          if (more && active(w_next, i)) issue_s(j + 1, i);
        }
        if (leader && ok && more) fa_mma_commit(bar_addr(sb, BAR_KEMPTY + (j + 1) % NSTAGE));
        w = w_next;
      }
    }
  } else if (warp < NSOFT) {
    // ================================ softmax warpgroups ==================================
    fa_setmaxnreg_inc<REGS_SOFTMAX>();
    const int i = warp >> 2;                       // query tile of this warpgroup
    const int lane_base = (warp & 3) * 32;         // TMEM lanes this warp may touch
    const int r = lane_base + lane;                // row inside the tile
    const int qi = DECODE ? (r & 63) : m0 + i * BM + r;  // query index
    const int half = DECODE ? (r >> 6) : 0;               // decode variant: kv columns 64 * half .. + 63 of every tile
    // decode variant: warps whose 32 rows are all padding (fewer than 33 queries) only keep the barrier protocol going
    const bool warp_active = !DECODE || (lane_base & 63) < p.Sq;
    fa_u32 idle_cnt = 0;
    const fa_u32 t_s = tmem + ((fa_u32)lane_base << 16) + COL_S + i * S_STRIDE;
    const fa_u32 t_o = tmem + ((fa_u32)lane_base << 16) + COL_O + i * D;
    const fa_u32 t_p = DECODE ? tmem + ((fa_u32)lane_base << 16) + COL_P + i * 64 : t_s;
    bool ok = true;
    // (rows beyond Sq have no row in the bit matrix: their scores are never stored, the mask is evaluated)
    const unsigned* rowbits = (p.t.mask_bits != nullptr && qi < p.Sq && (p.t.mask_hold == nullptr || *p.t.mask_hold != 0))
        ? p.t.mask_bits + (((long long)(p.t.mask_B == 1 ? 0 : b) * p.t.mask_H + (p.t.mask_H == 1 ? 0 : h)) * p.t.mask_rows + qi) * p.t.mask_stride
        : nullptr;
    SoftmaxCtx c = {p, sb, t_s, t_o, t_p, i, warp, qi, gb, gh, half, p.scale * FA_LOG2E, abort_flag, FA_NEG_INF, 0.f, 0u, rowbits, {}};
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE) && defined(FA_SCORE_LINEAR_KV)
    {
      const float mul = fa_score_mul(0.f, gb, gh, qi, 0) * c.sc2, slope = fa_score_add2_dkv(0.f, gb, gh, qi, 0);
      c.lin.m2 = fa_f2(mul, mul);
      c.lin.d = slope;
      for (int e = 0; e < 4; ++e) c.lin.od[e] = fa_f2(2 * e * slope, (2 * e + 1) * slope);
    }
#endif
    if (DECODE) {
      // the P columns of the other half of this lane's kv columns are never written again
      fa_u32 z[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) z[e] = 0u;
      fa_tmem_st16(t_p + (1 - half) * 32, z);
      fa_tmem_st16(t_p + (1 - half) * 32 + 16, z);
      fa_tmem_wait_st();
    }
#if FA_DTYPE == FA_DT_F32
    float acc[D];
#pragma unroll
    for (int e = 0; e < D; ++e) acc[e] = 0.f;
#endif
    // (the schedule entry of a step is read during the one before)
    fa_u32 w_next = sched[DECODE ? i : 0];
    for (int j = 0; j < nsteps && ok; ++j) {
      const fa_u32 w = w_next;
      w_next = sched[DECODE ? min(2 * j + 2 + i, MAXT) : j + 1];
      const int mode = DECODE ? (int)(w >> 16) : (int)((w >> (16 + 8 * i)) & 0xffu);
      const int tile = (int)(w & 0xffffu);
      if (mode == 0) continue;
      if (!warp_active) {
        // in step with the working warps: S of this step is there, then both arrivals they also make
        ok = fa_mbar_wait_warp(bar_addr(sb, BAR_S + i), idle_cnt & 1u, abort_flag);
        // The PV product of the previous step must be complete before this warp arrives on the P
        // barrier again: otherwise its arrival would be counted into the previous phase, which the
        // working warps may not have reached yet, and that product would start on unwritten P.
        if (ok && idle_cnt > 0) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_O + i), (idle_cnt - 1) & 1u, abort_flag);
        if (!ok) break;
        fa_tc_fence_after();
        fa_tc_fence_before();
        if (DECODE) fa_mbar_arrive(bar_addr(sb, BAR_SFREE2 + i));
        fa_mbar_arrive(bar_addr(sb, BAR_P + i));
        ++idle_cnt;
        continue;
      }
      const bool masked = (FA_HAS_MASK_MOD && mode == 1) || tile * BN + BN > p.Skv;
#if FA_DTYPE == FA_DT_F32
      ok = softmax_step_f32(c, acc, tile, mode, masked);
      continue;
#endif
      if (D == 64) ok = softmax_step<2>(c, tile, mode, masked);
      else ok = masked ? softmax_step<1>(c, tile, mode, true) : softmax_step<0>(c, tile, mode, false);
    }
    const float m_ref = c.m_ref, l = c.l;
    const fa_u32 cnt = warp_active ? c.cnt : idle_cnt;
    // ---- epilogue: O / l and the logsumexp of this thread's row ---------------------------
    if (ok && cnt > 0)
      ok = fa_mbar_wait_warp(bar_addr(sb, BAR_O + i + (ROT ? 2 * (int)((cnt - 1) & 1u) : 0)), (ROT ? (cnt - 1) >> 1 : cnt - 1) & 1u, abort_flag);
#if FA_TC_DECODE
    // The four partial results of a query row (two warpgroups x two column halves) are merged
    // inside the CTA: every thread puts its (O, maximum, sum) into shared memory, over the K / V
    // ring, which nothing reads or writes any more once both warpgroups have seen their last
    // product complete; then the 256 threads merge 64 rows x 64 columns and the CTA writes ONE
    // un-normalised partial result per row for the combine kernel.  All 256 softmax threads reach
    // both barriers, whatever happened before (every earlier wait is bounded).
    {
      constexpr int MP = D + 4;  // floats per scratch row: O[D], maximum, sum, pad (16-byte rows)
      float* scratch = (float*)(sm + OFF_K);
      static_assert(2 * 128 * MP * 4 <= 2 * NSTAGE * KV_STAGE, "merge scratch fits the K / V ring");
      asm volatile("bar.sync 2, 256;" ::: "memory");
      const bool good = ok && *abort_flag == 0;
      if (good && warp_active) {
        fa_tc_fence_after();
        float* row = scratch + (i * 128 + r) * MP;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          float o[32];
          if (cnt > 0) {
            fa_tmem_ld32(t_o + c * 32, o);
            fa_tmem_wait_ld();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = 0.f;
          }
#pragma unroll
          for (int e = 0; e < 32; e += 4) *(float4*)(row + c * 32 + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
        }
        *(float2*)(row + D) = make_float2(m_ref, m_ref != FA_NEG_INF ? l : 0.f);
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
      if (*abort_flag == 0) {
        const int mt = tid;                     // 0 .. 255
        const int mrow = mt >> 2, c0 = (mt & 3) * 16;  // query row, first of this thread's 16 columns
        if (mrow < p.Sq) {
          const float* src[4];
          float mm[4], mstar = FA_NEG_INF;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            src[k] = scratch + ((k >> 1) * 128 + (k & 1) * 64 + mrow) * MP;
            mm[k] = src[k][D];
            mstar = fmaxf(mstar, mm[k]);
          }
          float acc[16], lsum = 0.f;
#pragma unroll
          for (int e = 0; e < 16; ++e) acc[e] = 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float w = mm[k] == FA_NEG_INF ? 0.f : fa_ex2(mm[k] - mstar);
            lsum += w * src[k][D + 1];
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
              const float4 v4 = *(const float4*)(src[k] + c0 + e);
              acc[e] += w * v4.x; acc[e + 1] += w * v4.y; acc[e + 2] += w * v4.z; acc[e + 3] += w * v4.w;
            }
          }
          const long long prow = (((long long)b * p.Hq + h) * p.num_splits + split) * p.Sq + mrow;
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *(float4*)(p.part_o + prow * D + c0 + e) = make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]);
          if ((mt & 3) == 0) *(float2*)(p.part_ml + prow * 2) = make_float2(mstar, lsum);
        }
      }
    }
#else
    {
      // The output tile leaves through the shared memory of this warpgroup's query tile, which
      // nothing reads any more (every S product of the tile is complete): each thread converts its
      // row into the layout of the tile (128-byte rows, 16-byte chunk k of row r at k ^ (r & 7)) and
      // one tensor-map store per 64 columns writes whole lines and clips the rows beyond Sq.  (Each
      // thread storing its own row to global memory costs 32 different lines per instruction.)
      // All four warps of the warpgroup reach the barrier below, whatever happened before: every
      // earlier wait is bounded.
      // (a tile without kv steps: nothing has waited for the load of the query tile yet)
      if (ok && cnt == 0) ok = fa_mbar_wait_warp(bar_addr(sb, BAR_Q), 0, abort_flag);
      if (ok) {
        fa_tc_fence_after();
        // a row that never saw an unmasked key has no mass (its sum may hold the tiny values the
        // polynomial exponential returns for -inf): its output is 0
        const float inv = (l > 0.f && m_ref != FA_NEG_INF) ? 1.f / l : 0.f;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          float o[32];
          if (cnt > 0) {
            fa_tmem_ld32(t_o + c * 32, o);
            fa_tmem_wait_ld();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = 0.f;
          }
#if FA_DTYPE == FA_DT_F32
          {
            // 32 fp32 columns are one 128-byte row of a 128 x 128-byte block
            unsigned char* strow = sm + (i * ATOMS + c) * ATOM_BYTES + r * 128;
#pragma unroll
            for (int e = 0; e < 32; e += 4)
              *(float4*)(strow + (((e >> 2) ^ (r & 7)) * 16)) = make_float4((acc[32 * c + e] + o[e]) * inv, (acc[32 * c + e + 1] + o[e + 1]) * inv,
                                                                                 (acc[32 * c + e + 2] + o[e + 2]) * inv, (acc[32 * c + e + 3] + o[e + 3]) * inv);
            continue;
          }
#endif
          unsigned char* strow = sm + (i * ATOMS + (c >> 1)) * ATOM_BYTES + r * 128;
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 w;
            w.x = fa_pack2<DT>(o[e] * inv, o[e + 1] * inv);
            w.y = fa_pack2<DT>(o[e + 2] * inv, o[e + 3] * inv);
            w.z = fa_pack2<DT>(o[e + 4] * inv, o[e + 5] * inv);
            w.w = fa_pack2<DT>(o[e + 6] * inv, o[e + 7] * inv);
            *(uint4*)(strow + ((((c & 1) * 4 + (e >> 3)) ^ (r & 7)) * 16)) = w;
          }
        }
        if (p.lse != nullptr && qi < p.Sq)
          p.lse[((long long)b * p.Hq + h) * p.Sq + qi] = (l > 0.f && m_ref != FA_NEG_INF) ? (m_ref + (F32 ? log2f(l) : fa_lg2(l))) * FA_LN2 : FA_NEG_INF;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("bar.sync %0, 128;" ::"r"(3 + i) : "memory");
      if ((warp & 3) == 0 && lane == 0 && *abort_flag == 0 && m0 + i * BM < p.Sq) {
        // (a 128-byte column group of the output: 64 values of a 16-bit type, 32 of fp32)
        for (int a = 0; a < (F32 ? D / 32 : D / 64); ++a)
          fa_tma_store_4d(&P.to, sb + (i * ATOMS + a) * ATOM_BYTES, a * (F32 ? 32 : 64), m0 + i * BM, h, b);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tile must outlive the reads of the store
      }
    }
#endif
  }

  // ---- teardown ----------------------------------------------------------------------------
  fa_tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    fa_tc_fence_after();
    fa_tmem_dealloc(tmem, TMEM_COLS);
  }
  if (tid == 0 && *abort_flag != 0 && p.status != nullptr) atomicOr(p.status, FA_STATUS_WAIT_TIMEOUT);
}
