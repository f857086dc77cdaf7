// What the tcgen05 backward kernels share: launch parameters, small PTX helpers, the order of the items, the
// list of the pairs of one, and the masks read from the bit matrix.
#pragma once
#include "fa_sm100.cuh"

struct FaBwdTcParams {
  FaParams p;
  FaTensorMap tq, tk, tv, tdo;  // 4-d maps (D, S, H, B), 128-byte swizzle, box 64 x 128 rows
  FaTensorMap tdk, tdv;         // the outputs dK and dV, like tk and tv
  float* dq_acc;                // per (b, h, 128-row q tile): D / 32 fp32 blocks [128 rows][32 columns], 16-byte chunks of a row permuted
  const float* nlse2;           // [B, Hq, ceil(Sq/128)*128]: -lse * log2(e); -inf for rows without mass / beyond Sq
  const float* ndelta;          // same shape: -rowsum(O * dO); 0 beyond Sq
  int* work_counter;            // zero at launch: items beyond the first of every CTA are handed out through it
  int chunk_heads;              // (batch, kv head) pairs whose items are numbered together (see item_of)
};

namespace fa_bwd_items {

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void bulk_reduce_add_f32(float* gdst, fa_u32 ssrc, fa_u32 bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(gdst), "r"(ssrc), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// brings a tile into L2 ahead of the load that will need it
__device__ __forceinline__ void tma_prefetch_l2_4d(const FaTensorMap* map, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

// byte offset (in 16-byte units) of k-step kk of a K-major operand whose 64-element column groups
// are `atom_bytes` apart: 32 bytes per step inside a 128-byte row, four steps per group
__device__ __forceinline__ constexpr fa_u32 kstep_kmajor(int kk, int atom_bytes) {
  return (fa_u32)(((kk >> 2) * atom_bytes + (kk & 3) * 32) >> 4);
}

// Item number -> (kv head, batch, kv tile).  The first kv tiles of all heads come first (under a causal mask and
// with attention sinks they are the heaviest), then chunk by chunk of `ch` heads, in a chunk heads fastest and the
// kv tile slowest.  The CTAs work through the items in this order, so that at any time the dQ accumulator, Q and dO
// of about one chunk of heads are in use: the host sizes it to stay in L2.
struct Item {
  int hk, b, kt;
};
__device__ __forceinline__ Item item_of(int idx, int Hkv, int B, int n_kvt, int ch) {
  const unsigned heads = Hkv * B, i = idx;
  unsigned head = i, kt = 0;
  if ((unsigned)ch >= heads) {  // one chunk
    kt = i / heads;
    head = i - kt * heads;
  } else if (i >= heads) {
    const unsigned r = i - heads, per = ch * (n_kvt - 1), c = r / per, rr = r - c * per;
    const unsigned n = min((unsigned)ch, heads - c * ch);
    kt = rr / n;
    head = c * ch + rr - kt * n;
    ++kt;
  }
  const unsigned b = head / Hkv;
  return {(int)(head - b * Hkv), (int)b, (int)kt};
}

// The (query head, q tile) pairs of one item, written to `pl` by one warp: per head of the group,
// the 128-row q tiles the BlockMask lists for the item's kv tile (class 1: apply mask_mod, 2: full)
// in ascending order, one pair each.  Without tables every tile is listed.  Returns the
// number of pairs (the same in every lane).  `cl` is scratch: one bit per q tile and class.
template <int MAXPL, int MAXC>
__device__ __forceinline__ int build_pair_list(const FaParams& p, int hk, int b, int kt, int G, int n_ctiles,
                                               unsigned* cl, int* pl, int lane) {
  const bool tables = p.t.kv_num != nullptr && p.t.q_num != nullptr;
  int w = 0;
  for (int g = 0; g < G; ++g) {
    if (!tables) {
      const int nq = (p.Sq + 127) / 128;
      const int mode = FA_HAS_MASK_MOD ? 1 : 2;
      // the items of a head start at different q tiles, so that the CTAs on one head do not add to the same
      // dQ tile at the same time
      const int rot = kt % nq;
      for (int e = lane; e < nq && w + e < MAXPL; e += 32) pl[w + e] = (e + rot < nq ? e + rot : e + rot - nq) | (mode << 16) | (g << 20);
      w += nq;
      continue;
    }
    const int h = hk * G + g;
    if (lane < 2 * MAXC / 32) cl[lane] = 0u;
    __syncwarp();
    {
      // both counts are read before either index list (two round trips to memory, not four)
      const int bm = p.t.mB == 1 ? 0 : b, hm = p.t.mH == 1 ? 0 : h;
      const int kvblk = min(kt * 128 / p.t.KVB, p.t.nKV - 1);
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
          // (atomicOr on a generic address is 17 KB of code here, and its instruction-cache misses were paid by all warps)
          if (t < n_ctiles)
            asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(fa_smem_u32(cl + which * (MAXC / 32) + (t >> 5))), "r"(1u << (t & 31)) : "memory");
        }
        __syncwarp();
      }
    }
    for (int t0 = 0; t0 < n_ctiles; t0 += 32) {
      const int t = t0 + lane;
      // (only tiles below n_ctiles have a bit; a tile in both lists counts as full)
      const int c = (cl[MAXC / 32 + (t0 >> 5)] >> lane) & 1u ? 2 : (int)((cl[t0 >> 5] >> lane) & 1u);
      const unsigned listed = __ballot_sync(0xffffffffu, c != 0);
      const int at = w + __popc(listed & ((1u << lane) - 1u));
      if (c != 0 && at < MAXPL) pl[at] = t | (c << 16) | (g << 20);
      w += __popc(listed);
    }
    __syncwarp();
  }
  return min(w, MAXPL);
}

// Row `kv` of the transposed mask bit matrix (of its first (batch, head) entry), or null: not built, or out of date.
__device__ __forceinline__ const unsigned* bits_row(const FaParams& p, int kv) {
  const bool there = p.t.mask_bits_t != nullptr && (p.t.mask_hold == nullptr || *p.t.mask_hold != 0);
  return there ? p.t.mask_bits_t + (long long)kv * p.t.mask_t_stride : nullptr;
}
// Its words of q columns q0 .. q0+63, of entry (b, h)
__device__ __forceinline__ const unsigned* keep_words(const unsigned* bits, const FaParams& p, int b, int h, int q0) {
  const unsigned entry = (p.t.mask_B == 1 ? 0 : b) * p.t.mask_H + (p.t.mask_H == 1 ? 0 : h);
  return bits + (long long)entry * p.t.mask_t_rows * p.t.mask_t_stride + (q0 >> 5);
}
__device__ __forceinline__ void read_keep(fa_u32 (&keep)[2], const unsigned* bits, const FaParams& p, int b, int h, int q0) {
  const uint2 w = *(const uint2*)keep_words(bits, p, b, h, q0);
  keep[0] = w.x;
  keep[1] = w.y;
}
// The same if `want`, all ones else, for a pair that comes later: as one predicated instruction it leaves no branch behind whose end
// would wait for the load.
__device__ __forceinline__ void ask_keep(fa_u32 (&keep)[2], const unsigned* bits, const FaParams& p, int b, int h, int q0, bool want) {
  keep[0] = keep[1] = 0xffffffffu;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t}"
               : "+r"(keep[0]), "+r"(keep[1]) : "l"(keep_words(bits, p, b, h, q0)), "r"((int)(want && bits != nullptr)));
}
// Without a matrix (attention sink B1 H4 S32768, head dims 64 and 128, us: 695 -> 565, 785 -> 684; evaluated in line, in the
// first place: 659, 817): mask_mod of 32 columns at a time, from its range over them where that tells, else from a rolled loop over
// both words, which keeps the code small (unrolled over a thread's columns it is 64 copies of the user's mask).
__device__ __forceinline__ void eval_keep(fa_u32 (&keep)[2], int gb, int gh, int q0, int kv) {
#if FA_HAS_MASK_MOD
  int k0 = 1, k1 = 1;  // 0: none of the 32 columns, 2: all of them, 1: not known
#ifdef FA_HAS_MASK_RANGE
  k0 = fa_mask_range(gb, gh, q0, q0 + 31, kv, kv);
  k1 = fa_mask_range(gb, gh, q0 + 32, q0 + 63, kv, kv);
#endif
  fa_u32 w0 = 0u, w1 = 0u;
  if (k0 == 1 || k1 == 1) {
#pragma unroll 2
    for (int e = 0; e < 32; ++e) {
      w0 |= (fa_mask_mod(gb, gh, q0 + e, kv) ? 1u : 0u) << e;
      w1 |= (fa_mask_mod(gb, gh, q0 + 32 + e, kv) ? 1u : 0u) << e;
    }
  }
  keep[0] = k0 == 1 ? w0 : (k0 == 2 ? 0xffffffffu : 0u);
  keep[1] = k1 == 1 ? w1 : (k1 == 2 ? 0xffffffffu : 0u);
#endif
}
// Which of a thread's four steps of 16 columns have anything to compute: those in which a lane of its warp keeps a column (`masked`,
// the same for the warp), and none for a row beyond Skv.  At head dim 128, where the compute warps set the pace of a masked tile, this
// and asking for the words a pair ahead (ask_keep) took a pass over the long first items of an attention sink, B2 H16/4 S3001, from 345 to
// 314 us (pairs of 64 query rows: 310).  At head dim 64 it costs more than it saves (B2 H8 S8192 185 -> 195 us).
__device__ __forceinline__ fa_u32 live_steps(const fa_u32 (&keep)[2], bool masked, bool row_ok) {
  fa_u32 live = row_ok ? 0xfu : 0u;
  if (masked) {
    const fa_u32 a = __reduce_or_sync(0xffffffffu, row_ok ? keep[0] : 0u), b = __reduce_or_sync(0xffffffffu, row_ok ? keep[1] : 0u);
    live &= ((a & 0xffffu) ? 1u : 0u) | ((a >> 16) ? 2u : 0u) | ((b & 0xffffu) ? 4u : 0u) | ((b >> 16) ? 8u : 0u);
  }
  return live;
}
// Query columns beyond Sq have zero rows of Q and dO and a row scalar of -infinity, and a probability of zero with that, unless a
// score_mod is not finite there (score / (Sq - q)): then their keep bits have to go, on tiles of every kind.
#if FA_HAS_SCORE_MOD && !defined(FA_SCORE_FINITE_AT_0)
#define FA_BWD_CLEAR_BEYOND 1
#else
#define FA_BWD_CLEAR_BEYOND 0
#endif
#define FA_BWD_MASKS (FA_HAS_MASK_MOD || FA_BWD_CLEAR_BEYOND)  // some pairs are masked
// clears the bits of columns from `left` on (the number of columns below Sq); false: there are none
__device__ __forceinline__ bool clear_beyond(fa_u32 (&keep)[2], int left) {
  if (!FA_BWD_CLEAR_BEYOND || left >= 64) return false;
  const unsigned long long in = left <= 0 ? 0ull : (1ull << left) - 1ull;
  keep[0] &= (fa_u32)in;
  keep[1] &= (fa_u32)(in >> 32);
  return true;
}
// Clears in 16 pairs of 16-bit values the columns whose bit of `w` is not set, for P^T and dS^T after packing (head dim 64): one AND
// per pair in a block that only masked tiles enter, so that the code of all others stays what it is without a mask.  (What the
// exponential gave for a masked position, infinity too, goes with it.  A select per element made the kernel 15-20 % slower under a
// plain causal mask: B2 H8 S4096 126 -> 151 us.)  prmt copies the sign bit of a byte over eight bits where a selector's fourth bit is
// set: of w << s these are bits 7 - s, 15 - s, 23 - s and 31 - s, so that seven shifts and one prmt per pair make all masks of a word
// (five instructions per pair before: attention sink B2 H8 S8192 186 -> 172 us a pass, packed documents B4 H8 S4096 99 -> 92).
__device__ __forceinline__ void mask_pairs(fa_u32* pp, fa_u32* ds, fa_u32 w) {
  fa_u32 a[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) a[s] = w << s;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int s = 7 - ((2 * e) & 7), k = (2 * e) >> 3;
    fa_u32 m;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(m) : "r"(a[s]), "r"(a[s - 1]), "r"(0xcc88 + 0x1111 * k));
    pp[e] &= m;
    ds[e] &= m;
  }
}

}  // namespace fa_bwd_items
