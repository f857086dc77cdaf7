// Split-KV decode kernel for short query blocks (Sq <= 64): the key/value range of one
// (batch, head) is cut into `num_splits` contiguous runs of tiles, one CTA each, so that a
// single (b, h) with a long KV cache still fills the GPU.  The reference has no such path:
// for Sq < 16 it pads the query to 16 rows and runs its forward kernel with one program per
// (b, h) (flaxattention/core/attention.py:269-273, :310-311).
//
// CTA = 4 warps arranged as RG row groups x CG column groups (RG = BM/16, CG = 4/RG).  All
// warps share the K/V tiles, which stream through shared memory by TMA (FA_TMA: up to 16 rows, head dim 64 or 128) or in
// 16-byte cp.async pieces; warp (rg, cg) owns query rows 16*rg.. and the cg-th slice of each kv tile and keeps its own
// running (max, sum, O).  The CG partial results are merged through shared memory at the
// end.  With one split the CTA then writes O and LSE.  With several, the CTAs of a tile of rows are a thread-block cluster
// and merge through each other's shared memory (up to FA_DECODE_MAX_CLUSTER splits, when the host launches them so),
// or write un-normalised (O, max, sum) to the workspace for a second kernel to combine.
//
// With grouped-query attention the G query heads of a kv head can share one CTA
// (FA_PACK_HEADS): its G * Sq query rows form one tile, row r belonging to head r / Sq and
// query r % Sq, so K and V of the kv head are read once instead of G times.  The mods see the
// head and query index of each row; the BlockMask walk is the one of the group's first head,
// which is why the host packs only when the tables do not depend on the head.
//
// Compile-time parameters (macros): FA_DTYPE (fp16 / bf16), FA_D, FA_DV, FA_BM (16, 32, 64),
// FA_BN (kv tile), FA_PACK_HEADS, FA_STAGES, FA_TMA.
#pragma once
#include "fa_sm100.cuh"

// ---- thread-block clusters: barrier over all threads, reads of another CTA's shared memory ----
// (not the .aligned forms: the loops in front of the barriers leave the threads of a warp one by one)
__device__ __forceinline__ void fa_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ fa_u32 fa_mapa(fa_u32 addr, int rank) {
  fa_u32 r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 fa_ld_cluster_f2(fa_u32 addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 fa_ld_cluster_f4(fa_u32 addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

#ifndef FA_PACK_HEADS
#define FA_PACK_HEADS 0
#endif
#ifndef FA_TWO_PARTS
#define FA_TWO_PARTS 0  // 9 to 16 rows: the second part of the probabilities as a second instruction
#endif
#ifndef FA_CLUSTER
#define FA_CLUSTER 0  // the splits of a tile of rows are launched as a cluster (a variant of its own: with the merge in the kernel of
#endif                // all calls those without it took up to 7 % more, B16 H16 Skv1024 D64 16 rows 17.4 -> 18.6 us)

#ifndef FA_STAGES
#define FA_STAGES 2  // buffers of K and of V
#endif
#ifndef FA_TMA
#define FA_TMA 0  // K and V by TMA (see below)
#endif

struct FaDecodeParams {
  FaParams p;
#if FA_TMA
  FaTensorMap tk, tv;  // 4-d maps (D, S, H, B), box 64 x FA_BN / 4 x 1 x 1, 128-byte swizzle
#endif
};

namespace fa_dec {

constexpr bool PACK = FA_PACK_HEADS != 0;

constexpr int DT = FA_DTYPE;
constexpr int D = FA_D;
constexpr int DV = FA_DV;
constexpr int BM = FA_BM;
constexpr int BN = FA_BN;
constexpr int STAGES = FA_STAGES;
constexpr int NWARPS = 4;
constexpr int NT = NWARPS * 32;
constexpr int RG = BM / 16;
constexpr int CG = NWARPS / RG;
constexpr int WN = BN / CG;  // kv columns per warp and tile
constexpr int ES = 2;
constexpr int PQ = FaTile<D, ES>::PITCH;
constexpr int PV = FaTile<DV, ES>::PITCH;
// K and V by TMA (up to 16 rows, head dim 64 or 128): a warp's lane 0 asks for the WN keys of a tile that the warp reads, 64
// columns at a time, into buffers of the warp's own with barriers of their own.  Over seconds the pass is bound by power: 1000 W at
// 1.52 GHz with 16-byte cp.async copies, whose requests alone (no products, no softmax) kept B32 H8 Skv16384 D64 at 177 us, where
// bulk copies of the same bytes take 148.  us in a loop of seconds, cp.async / TMA / TMA and the splits that go with it: that call
// 185 / 165 / 158, 16 rows 195 / 176 / 171, B16 H32/8 Skv8191 D128 96 / 88 / 85; B8 H8 Skv2048 10.0 / 9.2 / 9.2.
constexpr bool TMA = FA_TMA != 0;
constexpr int ATOMS = D / 64;                      // 128-byte column groups of a row
constexpr int WBUF = WN * 128 * ATOMS;             // a warp's part of a tile of K or V
constexpr int Q_BYTES = BM * PQ;
constexpr int K_BYTES = TMA ? NWARPS * WBUF : BN * PQ;
constexpr int V_BYTES = TMA ? NWARPS * WBUF : BN * PV;
constexpr int MRG_PITCH = DV + 4;  // floats per merged row: O[DV], m, l, pad
constexpr int MRG_BYTES = CG * BM * MRG_PITCH * 4;
constexpr int PIPE_BYTES = STAGES * (K_BYTES + V_BYTES);
constexpr int BAR_BYTES = TMA ? (NWARPS * STAGES * 2 + 1) * 8 : 0;  // full barriers of K and V per warp and buffer; a flag
constexpr int PIPE_SPAN = PIPE_BYTES > MRG_BYTES ? PIPE_BYTES : MRG_BYTES;
constexpr int SMEM_BYTES = Q_BYTES + PIPE_SPAN + BAR_BYTES + (TMA ? 1024 : 0);  // (buffers at 1024 bytes)
// With one row group the probabilities go into P.V in two parts, rounded and what the rounding left.  One part alone has no error
// where a probability is exactly 1, at a running maximum, so that the fewer of these (fewer splits) the worse the results:
// B16 H32/8 Skv8191 D128 bf16, relative error against 64 bits, 2.11e-3 with three splits, 2.20e-3 with two, 1.66e-3 in two parts, nearly all
// of it the rounding of the output.  Up to 8 rows the second part lies in the 8 rows of the instruction that hold no query
// and costs nothing; up to 16 it takes a second instruction (FA_TWO_PARTS; B3 H16 Skv4096 D128, 16 rows: 28.3 us, 28.7 without), which
// the host asks for but where the tcgen05 kernel could run too: there one part is as good as that one (B8 H8 Skv8192 D64, 16 rows, bf16: error
// 2.18e-3 against 2.32e-3), and the second instruction costs time (34.3 us, 31.5 without).
constexpr bool TWO_PARTS = RG == 1;

// CTAs that share an SM by their shared memory: the registers must not allow fewer, up to three (170 registers), four (128) for two row
// groups of short rows (24 rows, B32 H8 Skv4096 D 16: 31.9 us with four, 45.3 with three, D 32 likewise; D 80 wants three for short
// caches).  Not with four row groups, whose warps need them (48 rows, B32 H8 Skv4096 D 32: 69 without, 78.6 with).
constexpr int SMEM_CTAS = 228 * 1024 / (SMEM_BYTES + 1024), MOST_CTAS = RG == 4 ? 1 : (RG == 2 && D + DV <= 64 ? 4 : 3);
constexpr int MIN_CTAS = SMEM_CTAS < MOST_CTAS ? (SMEM_CTAS > 0 ? SMEM_CTAS : 1) : MOST_CTAS;

static_assert(!TMA || (RG == 1 && D == DV && D % 64 == 0 && WN % 8 == 0), "TMA: warps on their own, whole column groups");
static_assert(DT != FA_DT_F32, "the decode kernel takes 16-bit inputs");
static_assert(BM == 16 || BM == 32 || BM == 64, "BM must be 16, 32 or 64");
static_assert(WN % 16 == 0, "each warp needs at least 16 kv columns per tile");

// The products of a warp over its part of a tile as TMA leaves it: rows of 128 bytes, 16-byte chunk c of row r at c ^ (r & 7),
// one block of WN rows per 64 columns.
__device__ __forceinline__ void mma_nt_sw(float (&acc)[WN / 8][4], const fa_u32 (&a)[D / 16][4], fa_u32 sB, int lane) {
  const fa_u32 x = ((lane >> 3) & 1) ^ (lane & 7);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const fa_u32 at = sB + (kk >> 2) * (WN * 128) + ((lane >> 4) * 8 + (lane & 7)) * 128 + (((kk & 3) * 2) ^ x) * 16;
#pragma unroll
    for (int nj = 0; nj < WN / 16; ++nj) {
      fa_u32 r0, r1, r2, r3;
      fa_ldsm_x4(at + nj * 2048, r0, r1, r2, r3);
      fa_mma16816<DT>(acc[2 * nj], a[kk], r0, r1);
      fa_mma16816<DT>(acc[2 * nj + 1], a[kk], r2, r3);
    }
  }
}
// (TWO: what the rounding of P leaves as a second product, as in fa_mma_nn)
template <bool TWO>
__device__ __forceinline__ void mma_nn_sw(float (&out)[DV / 8][4], const float (&pacc)[WN / 8][4], fa_u32 sB, int lane) {
  const fa_u32 x = (lane >> 4) ^ (lane & 7);
#pragma unroll
  for (int kj = 0; kj < WN / 16; ++kj) {
    fa_u32 a[4], rest[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float(&v)[4] = pacc[2 * kj + (i >> 1)];
      a[i] = fa_pack2<DT>(v[(i & 1) * 2], v[(i & 1) * 2 + 1]);
      if (TWO) {
        float r0, r1;
        fa_rest2<DT>(v[(i & 1) * 2], v[(i & 1) * 2 + 1], r0, r1);
        rest[i] = fa_pack2<DT>(r0, r1);
      }
    }
    const fa_u32 row = sB + (kj * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * 128;
#pragma unroll
    for (int dj = 0; dj < DV / 16; ++dj) {
      fa_u32 r0, r1, r2, r3;
      fa_ldsm_x4_t(row + (dj >> 2) * (WN * 128) + (((dj & 3) * 2) ^ x) * 16, r0, r1, r2, r3);
      fa_mma16816<DT>(out[2 * dj], a, r0, r1);
      fa_mma16816<DT>(out[2 * dj + 1], a, r2, r3);
      if (TWO) {
        fa_mma16816<DT>(out[2 * dj], rest, r0, r1);
        fa_mma16816<DT>(out[2 * dj + 1], rest, r2, r3);
      }
    }
  }
}

}  // namespace fa_dec

extern "C" __global__ void __launch_bounds__(fa_dec::NT, fa_dec::MIN_CTAS) fa_decode_kernel(const __grid_constant__ FaDecodeParams P) {
  using namespace fa_dec;
  const FaParams& p = P.p;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (TMA && (fa_dynamic_smem_size() < (fa_u32)SMEM_BYTES || blockDim.x != NT)) {
    // (a launch that does not fit the map: refused before anything is written)
    if (threadIdx.x == 0 && p.status != nullptr) atomicOr(p.status, FA_STATUS_BAD_LAUNCH);
    return;
  }
  // [buffers of K and V, later the rows to be merged | query tile | barriers]; without TMA the query tile lies in front
  unsigned char* const base = TMA ? smem_raw + ((1024u - (fa_smem_u32(smem_raw) & 1023u)) & 1023u) : smem_raw;
  unsigned char* const smem_q = TMA ? base + PIPE_SPAN : base;
  unsigned char* const smem_pipe = TMA ? base : base + Q_BYTES;
  FA_MOD_BUFS_INIT(p);
  fa_grid_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = warp % RG, cg = warp / RG;
  // grid: (splits, query heads, batch), or (splits, kv heads, batch) when the heads of a group are packed
  const int split = blockIdx.x, b = blockIdx.z;
  const int G = p.Hq / p.Hkv;
  const int hk = PACK ? (int)blockIdx.y : (int)blockIdx.y / G;
  const int h0 = PACK ? hk * G : (int)blockIdx.y;  // first query head of this CTA
  const int R = PACK ? G * p.Sq : p.Sq;            // query rows of this CTA
  const int gb = b + p.b_off;

  const fa_u32 sQ = fa_smem_u32(smem_q);
  const fa_u32 sK = fa_smem_u32(smem_pipe);
  const fa_u32 sV = sK + STAGES * K_BYTES;
#if FA_TMA
  const fa_u32 bars = sQ + Q_BYTES + warp * (STAGES * 16);  // this warp's: K 0 .. STAGES - 1, V 0 .. STAGES - 1
  volatile int* abort_flag = (volatile int*)(smem_q + Q_BYTES + NWARPS * STAGES * 16);
  if (tid == 0) {
    for (int i = 0; i < NWARPS * STAGES * 2; ++i) fa_mbar_init(sQ + Q_BYTES + i * 8, 1);
    fa_mbar_init_fence();
    *abort_flag = 0;
  }
  __syncthreads();
#endif

  const char* qg = (const char*)p.q.ptr + (long long)b * p.q.sb * ES;
  const char* kg = (const char*)p.k.ptr + ((long long)b * p.k.sb + (long long)hk * p.k.sh) * ES;
  const char* vg = (const char*)p.v.ptr + ((long long)b * p.v.sb + (long long)hk * p.v.sh) * ES;

  {
    // query tile: row r is query r % Sq of head h0 + r / Sq; rows from R on are zero-filled
    constexpr int CPR = D * ES / 16;
    for (int i = tid; i < BM * CPR; i += NT) {
      const int r = i / CPR, c = i - r * CPR;
      const bool ok = r < R;
      const int g = PACK ? r / p.Sq : 0, q = r - g * p.Sq;
      const char* src = qg + (ok ? ((long long)(h0 + g) * p.q.sh + (long long)q * p.q.ss) * ES + c * 16 : 0);
      fa_cp_async16(sQ + r * PQ + c * 16, src, ok ? 16 : 0);
    }
  }
  fa_cp_commit();

  FaWalk walk;
  walk.init_kv<BN>(p.t, b, h0, 0, p.Skv);
  // this split's run of tile slots, gone through block by block (without tables every tile is a block)
  const int per = (walk.total + p.num_splits - 1) / p.num_splits;
  const int slot0 = min(split * per, walk.total);
  int left = min(slot0 + per, walk.total) - slot0;  // slots still to be taken
  const bool tables = walk.idx[0] != nullptr;
  int block = !tables || walk.tpb == 1 ? slot0 : slot0 / walk.tpb, tile = tables ? slot0 - block * walk.tpb : 0;  // of the next slot
  // The table entry of a block is read when the last tile of the one before it is taken, a tile before its loads go out.
  // (Read when it is needed, it is a trip to L2 in front of every load: causal offset mask, B32 H8 Skv16384 D64, 1 row
  // 173 -> 168 us, 16 rows 184 -> 178.)
  int entry = walk.entry(block);
  auto next_tile = [&](int& n0, bool& full) -> bool {
    while (left > 0) {
      n0 = walk.start_of<BN>(block, tile, entry, full);
      --left;
      if (!tables || ++tile == walk.tpb) {
        tile = 0;
        ++block;
        entry = walk.entry(block);
      }
      if (n0 >= 0) return true;
    }
    return false;
  };
  // With one row group (Sq <= 16) every warp reads only its own WN keys of a tile: it then loads
  // just those rows itself and the warps run as independent pipelines, with no block-wide
  // barrier inside the kv loop.  With several row groups the tile is loaded cooperatively.
  constexpr bool PRIVATE = RG == 1;
#if FA_TMA
  auto load_tile = [&](const FaTensorMap* map, fa_u32 dst, fa_u32 bar, int n0) {
    if (lane == 0) {
      fa_mbar_expect_tx(bar, WBUF);
#pragma unroll
      for (int a = 0; a < ATOMS; ++a) fa_tma_load_4d(dst + a * (WN * 128), map, bar, a * 64, n0 + cg * WN, hk, b);
    }
  };
  auto load_k = [&](int stage, int n0) { load_tile(&P.tk, sK + stage * K_BYTES + cg * WBUF, bars + stage * 8, n0); };
  auto load_v = [&](int stage, int n0) { load_tile(&P.tv, sV + stage * V_BYTES + cg * WBUF, bars + (STAGES + stage) * 8, n0); };
#else
  auto load_k = [&](int stage, int n0) {
    if (PRIVATE) {
      const int first = n0 + cg * WN, vr = p.Skv - first;
      const long long koff = vr > 0 ? (long long)first * p.k.ss * ES : 0;
      fa_load_tile<D, ES, 32>(sK + stage * K_BYTES + cg * WN * PQ, kg + koff, p.k.ss * ES, WN, vr, lane);
    } else {
      fa_load_tile<D, ES, NT>(sK + stage * K_BYTES, kg + (long long)n0 * p.k.ss * ES, p.k.ss * ES, BN, p.Skv - n0, tid);
    }
  };
  auto load_v = [&](int stage, int n0) {
    if (PRIVATE) {
      const int first = n0 + cg * WN, vr = p.Skv - first;
      const long long voff = vr > 0 ? (long long)first * p.v.ss * ES : 0;
      fa_load_tile<DV, ES, 32>(sV + stage * V_BYTES + cg * WN * PV, vg + voff, p.v.ss * ES, WN, vr, lane);
    } else {
      fa_load_tile<DV, ES, NT>(sV + stage * V_BYTES, vg + (long long)n0 * p.v.ss * ES, p.v.ss * ES, BN, p.Skv - n0, tid);
    }
  };
#endif

  float o[DV / 8][4];
#pragma unroll
  for (int j = 0; j < DV / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m_run[2] = {FA_NEG_INF, FA_NEG_INF}, l_run[2] = {0.f, 0.f};

  // K and V are released and asked for separately: the K buffer of a tile is free as soon as its scores are
  // there, so K of the tile STAGES further on is under way during this tile's P.V, and V of the one STAGES - 1 further on
  // during its scores: STAGES - 1/2 tiles are always in flight (with both loads issued together at the top of the loop it
  // would be STAGES - 1).
  int n0_at[STAGES];       // this tile and the ones whose K has been asked for
  bool full_at[STAGES], have[STAGES];
#pragma unroll
  for (int t = 0; t < STAGES; ++t) {
    n0_at[t] = 0;
    full_at[t] = false;
    have[t] = (t == 0 || have[t > 0 ? t - 1 : 0]) && next_tile(n0_at[t], full_at[t]);
    if (have[t]) load_k(t, n0_at[t]);
    fa_cp_commit();
    if (t < STAGES - 1) {
      if (have[t]) load_v(t, n0_at[t]);
      fa_cp_commit();
    }
  }
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE) && defined(FA_SCORE_LINEAR_KV)
  // A bias that is linear over kv (ALiBi) under a multiplier that does not read it: multiplier and slope of this thread's two rows
  // are taken here, the bias once per tile at the thread's first key, and the other keys add multiples of the slope.  To the scores:
  // added to the bias, they would round a large one once more per key (60000 + kv / 2048: error of the probabilities 2.9e-3,
  // where three roundings are 2.7e-3).
  constexpr int LIN_KEPT = WN / 8 <= 4 ? WN / 8 : 0;  // (pairs of multiples in registers)
  fa_u64 lin_m[2], lin_d[2], lin_od[2][LIN_KEPT > 0 ? LIN_KEPT : 1];
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int row = rg * 16 + hh * 8 + (lane >> 2);
    const int g_row = PACK ? row / p.Sq : 0;
    const int qi = row - g_row * p.Sq, gh = h0 + g_row + p.h_off;
    const float mul = fa_score_mul(0.f, gb, gh, qi, 0) * (p.scale * FA_LOG2E), slope = fa_score_add2_dkv(0.f, gb, gh, qi, 0);
    lin_m[hh] = fa_f2(mul, mul);
    lin_d[hh] = fa_f2(slope, slope);
#pragma unroll
    for (int j = 0; j < LIN_KEPT; ++j) lin_od[hh][j] = fa_f2((float)(j * 8) * slope, (float)(j * 8 + 1) * slope);
  }
#endif
  fa_u32 qf[D / 16][4];
  bool q_loaded = false;
  int cur = 0;  // buffer of the tile being computed
  [[maybe_unused]] fa_u32 phase = 0;
#if FA_TMA
  fa_cp_wait<0>();
  __syncthreads();  // the query tile
#endif

  while (have[0]) {
#if FA_TMA
    if (!fa_mbar_wait_all(bars + cur * 8, phase, abort_flag)) break;  // K of this tile
#else
    fa_cp_wait<2 * (STAGES - 1)>();  // K of this tile (what was asked for after it may still be on its way)
    if (PRIVATE && q_loaded) __syncwarp();
    else __syncthreads();  // (first iteration: the query tile was loaded by all threads)
#endif
    if (have[STAGES - 1]) load_v(cur == 0 ? STAGES - 1 : cur - 1, n0_at[STAGES - 1]);
    fa_cp_commit();

    if (!q_loaded) {
      q_loaded = true;
      fa_load_a_frags<D>(qf, sQ, PQ, rg * 16, lane);
    }
    const int n0 = n0_at[0] + cg * WN;
    const bool full = full_at[0];
    float s[WN / 8][4];
#pragma unroll
    for (int j = 0; j < WN / 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#if FA_TMA
    mma_nt_sw(s, qf, sK + cur * K_BYTES + cg * WBUF, lane);
#else
    fa_mma_nt<DT, D, WN>(s, qf, sK + cur * K_BYTES + cg * WN * PQ, PQ, lane);
#endif

    fa_round_acc<DT, WN / 8>(s);
    const bool ragged = n0 + WN > p.Skv;
    const float sc2 = p.scale * FA_LOG2E;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      // rows 8..15 of a row group hold no query when there are at most 8 (+ 16 rg) rows: nothing to do for them
      if (rg * 16 + hh * 8 >= R) {
#pragma unroll
        for (int j = 0; j < WN / 8; ++j) {
          // (hh = 1, TWO_PARTS: the second part of the rows 8 above)
          if (TWO_PARTS) fa_rest2<DT>(s[j][0], s[j][1], s[j][2], s[j][3]);
          else s[j][hh * 2] = s[j][hh * 2 + 1] = 0.f;
        }
        continue;
      }
      const int row = rg * 16 + hh * 8 + (lane >> 2);
      const int g_row = PACK ? row / p.Sq : 0;
      const int qi = row - g_row * p.Sq;
      const int gh = h0 + g_row + p.h_off;
      const int kv0 = n0 + (lane & 3) * 2;  // first key of this thread
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE) && defined(FA_SCORE_LINEAR_KV)
      const float bias0 = fa_score_add2(0.f, gb, gh, qi, kv0);
      const fa_u64 lin_b = fa_f2(bias0, bias0);
#endif
#pragma unroll
      for (int j = 0; j < WN / 8; ++j) {
        const int kv = kv0 + j * 8;
        float x0 = s[j][hh * 2], x1 = s[j][hh * 2 + 1];
#if FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE) && defined(FA_SCORE_LINEAR_KV)
        const fa_u64 od = LIN_KEPT > 0 ? lin_od[hh][LIN_KEPT > 0 ? j : 0] : fa_mul2(fa_f2((float)(j * 8), (float)(j * 8 + 1)), lin_d[hh]);
        fa_f2_unpack(fa_add2(fa_fma2(fa_f2(x0, x1), lin_m[hh], od), lin_b), x0, x1);
#elif FA_HAS_SCORE_MOD && defined(FA_SCORE_AFFINE)
        // affine score_mod: scale and log2(e) folded into one FMA
        x0 = fmaf(x0, fa_score_mul(0.f, gb, gh, qi, kv) * sc2, fa_score_add2(0.f, gb, gh, qi, kv));
        x1 = fmaf(x1, fa_score_mul(0.f, gb, gh, qi, kv + 1) * sc2, fa_score_add2(0.f, gb, gh, qi, kv + 1));
#elif FA_HAS_SCORE_MOD
        x0 = fa_score_mod(x0 * p.scale, gb, gh, qi, kv) * FA_LOG2E;
        x1 = fa_score_mod(x1 * p.scale, gb, gh, qi, kv + 1) * FA_LOG2E;
#else
        x0 *= sc2;
        x1 *= sc2;
#endif
        s[j][hh * 2] = x0;
        s[j][hh * 2 + 1] = x1;
      }
      if (ragged || (FA_HAS_MASK_MOD && !full)) {
#pragma unroll
        for (int j = 0; j < WN / 8; ++j) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int kv = kv0 + j * 8 + e;
            bool keep = kv < p.Skv;
#if FA_HAS_MASK_MOD
            if (!full) keep = keep && fa_mask_mod(gb, gh, qi, kv);
#endif
            if (!keep) s[j][hh * 2 + e] = FA_NEG_INF;
          }
        }
      }
      float mx = FA_NEG_INF;
#pragma unroll
      for (int j = 0; j < WN / 8; ++j) mx = fa_max3(mx, s[j][hh * 2], s[j][hh * 2 + 1]);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run[hh], mx);
      const float m_use = (m_new == FA_NEG_INF) ? 0.f : m_new;
      const float corr = fa_ex2(m_run[hh] - m_use);
      m_run[hh] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < WN / 8; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float pv = fa_ex2(s[j][hh * 2 + e] - m_use);
          s[j][hh * 2 + e] = pv;
          sum += pv;
        }
      }
      l_run[hh] = l_run[hh] * corr + sum;
      // (after the first tiles the maximum seldom moves)
      if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
        for (int j = 0; j < DV / 8; ++j) {
          o[j][hh * 2] *= corr;
          o[j][hh * 2 + 1] *= corr;
          if (TWO_PARTS && R <= 8) {
            o[j][2] *= corr;
            o[j][3] *= corr;
          }
        }
      }
    }
#if FA_TMA
    if (!fa_mbar_wait_all(bars + (STAGES + cur) * 8, phase, abort_flag)) break;  // V of this tile
    __syncwarp();
#else
    fa_cp_wait<2 * (STAGES - 1)>();  // V of this tile
    if (PRIVATE) __syncwarp();
    else __syncthreads();
#endif
#pragma unroll
    for (int t = 0; t + 1 < STAGES; ++t) {
      have[t] = have[t + 1];
      n0_at[t] = n0_at[t + 1];
      full_at[t] = full_at[t + 1];
    }
    have[STAGES - 1] = have[STAGES - 1] && next_tile(n0_at[STAGES - 1], full_at[STAGES - 1]);
    if (have[STAGES - 1]) load_k(cur, n0_at[STAGES - 1]);
    fa_cp_commit();
#if FA_TMA
    if (TWO_PARTS && FA_TWO_PARTS && R > 8) mma_nn_sw<true>(o, s, sV + cur * V_BYTES + cg * WBUF, lane);
    else mma_nn_sw<false>(o, s, sV + cur * V_BYTES + cg * WBUF, lane);
    __syncwarp();  // (every lane has read V before its buffer is asked for again)
#else
    if (TWO_PARTS && FA_TWO_PARTS && R > 8) fa_mma_nn<DT, WN, DV, true>(o, s, sV + cur * V_BYTES + cg * WN * PV, PV, lane);
    else fa_mma_nn<DT, WN, DV>(o, s, sV + cur * V_BYTES + cg * WN * PV, PV, lane);
#endif
    if (++cur == STAGES) {
      cur = 0;
      phase ^= 1u;
    }
  }

  fa_grid_release();
  // ---- merge the CG column groups ------------------------------------------------------
  fa_cp_wait<0>();
  __syncthreads();
  float* mrg = (float*)smem_pipe;
  if (TWO_PARTS && R <= 8) {
#pragma unroll
    for (int j = 0; j < DV / 8; ++j) {
      o[j][0] += o[j][2];
      o[j][1] += o[j][3];
    }
  }
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    float l = l_run[hh];
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const int r = rg * 16 + hh * 8 + (lane >> 2);
    float* row = mrg + ((long long)cg * BM + r) * MRG_PITCH;
#pragma unroll
    for (int j = 0; j < DV / 8; ++j) {
      const int c = j * 8 + (lane & 3) * 2;
      row[c] = o[j][hh * 2];
      row[c + 1] = o[j][hh * 2 + 1];
    }
    if ((lane & 3) == 0) {
      row[DV] = m_run[hh];
      row[DV + 1] = l;
    }
  }
  __syncthreads();
  const int rows = min(R, BM);
  // Splits in one cluster: the CTA's merged rows stay in shared memory, O over the first column group's and the
  // maximum and sum over the query tile, and the CTAs of the cluster read each other's.
  constexpr bool in_cluster = FA_CLUSTER != 0;
  float2* ml = (float2*)smem_q;  // [BM]
  for (int i = tid; i < rows * DV; i += NT) {
    const int r = i / DV, c = i - r * DV;
    const int g_row = PACK ? r / p.Sq : 0, qr = r - g_row * p.Sq, h = h0 + g_row;
    const long long bh = (long long)b * p.Hq + h;
    float mstar = FA_NEG_INF;
#pragma unroll
    for (int g = 0; g < CG; ++g) mstar = fmaxf(mstar, mrg[((long long)g * BM + r) * MRG_PITCH + DV]);
    float acc = 0.f, lstar = 0.f;
#pragma unroll
    for (int g = 0; g < CG; ++g) {
      const float* row = mrg + ((long long)g * BM + r) * MRG_PITCH;
      const float w = row[DV] == FA_NEG_INF ? 0.f : fa_ex2(row[DV] - mstar);
      acc += w * row[c];
      lstar += w * row[DV + 1];
    }
    if (in_cluster) {
      mrg[(long long)r * MRG_PITCH + c] = acc;  // (this thread alone reads column c of the row)
      if (c == 0) ml[r] = make_float2(mstar, lstar);
    } else if (p.num_splits > 1) {
      const long long prow = (bh * p.num_splits + split) * p.Sq + qr;
      p.part_o[prow * DV + c] = acc;
      if (c == 0) {
        p.part_ml[prow * 2] = mstar;
        p.part_ml[prow * 2 + 1] = lstar;
      }
    } else {
      const float inv = lstar > 0.f ? 1.f / lstar : 0.f;
      char* og = (char*)p.o.ptr + ((long long)b * p.o.sb + (long long)h * p.o.sh + (long long)qr * p.o.ss) * ES;
      const float val = acc * inv;
      if (DT == FA_DT_F16) {
        fa_u16 hv;
        asm("cvt.rn.f16.f32 %0, %1;" : "=h"(hv) : "f"(val));
        ((fa_u16*)og)[c] = hv;
      } else {
        fa_u16 hv;
        asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(hv) : "f"(val));
        ((fa_u16*)og)[c] = hv;
      }
      // (log2f, as in the merges, takes 1.5 us of 34 with 64 rows: B16 H16 Skv1024 D64)
      if (c == 0 && p.lse != nullptr)
        p.lse[bh * p.Sq + qr] = lstar > 0.f ? (mstar + (RG == 1 ? log2f(lstar) : fa_lg2(lstar))) * FA_LN2 : FA_NEG_INF;
    }
  }
#if FA_CLUSTER
  // ---- merge the splits: four columns of a row per thread, the rows spread over the CTAs -----------
  fa_cluster_sync();
  const int ns = p.num_splits;
  for (int i = split * NT + tid; i < rows * (DV / 4); i += ns * NT) {
    const int r = i / (DV / 4), c = (i - r * (DV / 4)) * 4;
    const int g_row = PACK ? r / p.Sq : 0, qr = r - g_row * p.Sq, h = h0 + g_row;
    const fa_u32 ml_addr = fa_smem_u32(ml + r), o_addr = fa_smem_u32(mrg + (long long)r * MRG_PITCH + c);
    float2 part[FA_DECODE_MAX_CLUSTER];
    float mstar = FA_NEG_INF;
#pragma unroll
    for (int s = 0; s < FA_DECODE_MAX_CLUSTER; ++s) {
      part[s] = s < ns ? fa_ld_cluster_f2(fa_mapa(ml_addr, s)) : make_float2(FA_NEG_INF, 0.f);
      mstar = fmaxf(mstar, part[s].x);
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float lstar = 0.f;
#pragma unroll
    for (int s = 0; s < FA_DECODE_MAX_CLUSTER; ++s) {
      const float w = part[s].x == FA_NEG_INF ? 0.f : exp2f(part[s].x - mstar);
      if (w == 0.f) continue;
      const float4 x = fa_ld_cluster_f4(fa_mapa(o_addr, s));
      acc.x += w * x.x; acc.y += w * x.y; acc.z += w * x.z; acc.w += w * x.w;
      lstar += w * part[s].y;
    }
    const float inv = lstar > 0.f ? 1.f / lstar : 0.f;
    char* og = (char*)p.o.ptr + ((long long)b * p.o.sb + (long long)h * p.o.sh + (long long)qr * p.o.ss + c) * ES;
    *(uint2*)og = make_uint2(fa_pack2<DT>(acc.x * inv, acc.y * inv), fa_pack2<DT>(acc.z * inv, acc.w * inv));
    if (c == 0 && p.lse != nullptr)
      p.lse[((long long)b * p.Hq + h) * p.Sq + qr] = lstar > 0.f ? (mstar + log2f(lstar)) * FA_LN2 : FA_NEG_INF;
  }
  fa_cluster_sync();  // nobody leaves while its rows are being read
#endif
#if FA_TMA
  if (tid == 0 && *abort_flag != 0 && p.status != nullptr) atomicOr(p.status, FA_STATUS_WAIT_TIMEOUT);
#endif
}
