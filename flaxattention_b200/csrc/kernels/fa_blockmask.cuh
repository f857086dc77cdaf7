// mask_mod over a block grid, for create_block_mask.  Replaces the dense-mask route of
// flaxattention/core/blockmask.py:277-369 (create_mask -> reshape -> block sums): every position is
// evaluated once, the class of each block (0 = no position kept, 1 = some, 2 = all) comes from the
// counts, and the mask itself is kept as bit matrices (row-major and transposed) where the caller wants
// them; a dense [B,H,Q,KV] mask does not exist.
// Positions beyond Q_LEN / KV_LEN are classified like any other, because the reference classifies on
// the lengths rounded up to whole blocks (core/blockmask.py:440-444); in the bit matrices they are 0.
// The mod fragment (fa_mask_mod, FA_HAS_MASK_MOD) is placed before this file.
#pragma once
#include "fa_params.h"

// One CTA of eight warps per block, in 128 x 128 sub-tiles: a warp takes 32 rows and 64 keys, a lane one key out of each group of 32.
// A mask over captured tensors gets four warps of 32 rows and 128 keys: lane = key makes what it reads per key (a document id) a
// coalesced load outside the row loop, and what it reads per query is a broadcast that serves all groups (12 documents, 4096 x 4096:
// 8.6 us, with eight warps 10.5; others are bound by the time one warp takes: attention sink, 8192 x 8192, 10.1 against 11.1).
// The lane's own bits over the rows are a word of the transposed matrix (one predicated OR per position), and five exchange steps
// between the lanes turn the 32 words into those of the row-major one.  Both matrices and the block's count come out of one
// evaluation.  Where interval arithmetic over the mask's expression (fa_mask_range, from the tracer) says that a whole block, or
// 32 x 32 positions of it, are all kept or all not, none is evaluated; a whole block is constant words.
// Bound by the chain of a partial block's evaluation at the end of the grid, and by launches.  8192 x 8192 positions of an
// attention-sink mask, with the tables: 17.6 us (four warps per block, whole blocks put together like partial ones) -> 12.6.
// Lane = row instead took up to 1.6 times as long with masks that read by key (8192 x 8192, one id per key) and with few rows.
// Needs key blocks of whole 32-bit words and query blocks of whole words or a single one; other block sizes go to the
// classify kernel below.
#ifndef FA_SCAN_GROUPS
#define FA_SCAN_GROUPS 4  // groups of 32 keys of a warp
#endif
constexpr int FA_SCAN_WARPS = 16 / FA_SCAN_GROUPS;
// the transpose of the 32 x 32 bit matrix whose row i is lane i's word
__device__ __forceinline__ unsigned fa_bit_transpose(unsigned x, int lane) {
  unsigned m = 0x0000ffffu;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const unsigned y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? (x & ~m) | ((y & ~m) >> s) : (x & m) | ((y & m) << s);
    m ^= m << (s >> 1);
  }
  return x;
}
extern "C" __global__ void __launch_bounds__(32 * FA_SCAN_WARPS) fa_mask_scan_kernel(const __grid_constant__ FaMaskParams p) {
  FA_MOD_BUFS_INIT(p);
  fa_grid_wait();
  fa_grid_release();
  __shared__ __align__(16) unsigned t_words[128][4];
  __shared__ int s_cnt[FA_SCAN_WARPS];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvb = blockIdx.x, qb = blockIdx.y, bh = blockIdx.z;
  const int b = bh / p.H, h = bh - b * p.H;
  const int gb = b + p.b_off, gh = h + p.h_off;
  const int q0 = qb * p.QB, k0 = kvb * p.KVB;
  constexpr int G = FA_SCAN_GROUPS;
  int cnt = 0;
#ifdef FA_HAS_MASK_RANGE
  // A block of 128 x 128 inside both lengths that is all kept or all not: constant words, nothing to exchange.
  if (p.QB == 128 && p.KVB == 128 && q0 + 128 <= p.Q_LEN && k0 + 128 <= p.KV_LEN) {
    const int known = fa_mask_range(gb, gh, q0, q0 + 127, k0, k0 + 127);
    if (known != 1) {
      const unsigned w = known ? 0xffffffffu : 0u;
      const uint4 w4 = make_uint4(w, w, w, w);
      const int i = threadIdx.x & 127;
      if (threadIdx.x < 128 && p.bits != nullptr) *(uint4*)(p.bits + ((long long)bh * p.Q_LEN + q0 + i) * p.stride + (k0 >> 5)) = w4;
      if ((FA_SCAN_WARPS == 4 || threadIdx.x >= 128) && p.bits_t != nullptr) *(uint4*)(p.bits_t + ((long long)bh * p.KV_LEN + k0 + i) * p.stride_t + (q0 >> 5)) = w4;
      if (threadIdx.x == 0 && p.cls != nullptr) p.cls[((long long)bh * p.nQ + qb) * p.nKV + kvb] = (signed char)(known ? 2 : 0);
      return;
    }
  }
#endif
  for (int r0 = 0; r0 < p.QB; r0 += 128) {
    const int row = r0 + (warp & 3) * 32 + lane, q = q0 + row;  // the row of the block whose words this lane writes, and its query
    const int qw = q - lane, nrows = min(32, p.QB - (row - lane));  // first query of the warp, and how many it has
    for (int c0 = 0; c0 < p.KVB; c0 += 128) {
      const int cw = c0 + (warp >> 2) * 32 * G, k2 = k0 + cw;  // first key of the warp
      unsigned colw[G] = {};  // bit r: query qw + r, key k2 + 32 c + lane
      if (nrows >= 16) {  // (rows that the block does not have are evaluated with the others and dropped)
        int open = cw + 32 * G <= p.KVB ? (1 << G) - 1 : (cw < p.KVB ? (1 << ((p.KVB - cw + 31) / 32)) - 1 : 0);  // groups of 32 keys to evaluate (the same for the warp)
#ifdef FA_HAS_MASK_RANGE
#pragma unroll
        for (int c = 0; c < G; ++c) {
          const int known = (open >> c) & 1 ? fa_mask_range(gb, gh, qw, qw + 31, k2 + 32 * c, k2 + 32 * c + 31) : 1;
          if (known != 1) {
            open &= ~(1 << c);
            colw[c] = known ? 0xffffffffu : 0u;
          }
        }
#endif
        if (open == (1 << G) - 1) {
#pragma unroll 1
          for (int r = 0; r < 32; r += 8) {
            unsigned m[G] = {};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
#pragma unroll
              for (int c = 0; c < G; ++c)
                if (fa_mask_mod(gb, gh, qw + r + e, k2 + 32 * c + lane)) m[c] |= 1u << e;
            }
#pragma unroll
            for (int c = 0; c < G; ++c) colw[c] |= m[c] << r;
          }
        } else {
#pragma unroll 1
          for (; open != 0; open &= open - 1) {
            const int c1 = __ffs(open) - 1;
            unsigned w = 0u;
#pragma unroll 1
            for (int r = 0; r < 32; r += 8) {
              unsigned m = 0u;
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (fa_mask_mod(gb, gh, qw + r + e, k2 + 32 * c1 + lane)) m |= 1u << e;
              w |= m << r;
            }
#pragma unroll
            for (int c = 0; c < G; ++c) colw[c] = c == c1 ? w : colw[c];
          }
        }
      } else {
#pragma unroll 1
        for (int r = 0; r < nrows; ++r) {
#pragma unroll
          for (int c = 0; c < G; ++c)
            if (fa_mask_mod(gb, gh, qw + r, k2 + 32 * c + lane)) colw[c] |= 1u << r;
        }
      }
#pragma unroll
      for (int c = 0; c < G; ++c) {
        if (cw + 32 * c + lane >= p.KVB) colw[c] = 0u;
        if (nrows < 32) colw[c] &= (1u << max(nrows, 0)) - 1u;
        cnt += __popc(colw[c]);
        if (p.bits_t != nullptr) t_words[cw - c0 + 32 * c + lane][warp & 3] = colw[c];
      }
      if (p.bits != nullptr) {
        // the row's words of this warp's keys; keys beyond KV_LEN are 0, and the last block also writes the padding words
        unsigned roww[G];
#pragma unroll
        for (int c = 0; c < G; ++c) {
          const int left = p.KV_LEN - (k2 + 32 * c);
          roww[c] = fa_bit_transpose(colw[c], lane);
          if (left < 32) roww[c] &= left <= 0 ? 0u : (1u << left) - 1u;
        }
        if (row < p.QB && q < p.Q_LEN) {
          unsigned* dst = p.bits + ((long long)bh * p.Q_LEN + q) * p.stride;
          const int w0 = k2 >> 5;
          const bool last = kvb == p.nKV - 1 && c0 + 128 >= p.KVB;  // (the padding lies behind the last warps' words)
          const int wend = last ? ((warp >> 2) == FA_SCAN_WARPS / 4 - 1 ? (int)p.stride : min(w0 + G, (int)p.stride)) : min(w0 + G, (k0 + p.KVB) >> 5);
          if (G == 4 && (w0 & 3) == 0 && w0 + 4 <= wend) {
            *(uint4*)(dst + w0) = make_uint4(roww[0], roww[1], roww[G - 2], roww[G - 1]);
          } else if (G == 2 && (w0 & 1) == 0 && w0 + 2 <= wend) {
            *(uint2*)(dst + w0) = make_uint2(roww[0], roww[1]);
          } else {
#pragma unroll
            for (int c = 0; c < G; ++c)
              if (w0 + c < wend) dst[w0 + c] = roww[c];
          }
          for (int w = w0 + G; w < wend; ++w) dst[w] = 0u;
        }
      }
      if (p.bits_t != nullptr) {
        __syncthreads();
        const int col = c0 + (int)threadIdx.x, kv = k0 + col;
        if (threadIdx.x < 128 && col < p.KVB && kv < p.KV_LEN) {
          unsigned* dst = p.bits_t + ((long long)bh * p.KV_LEN + kv) * p.stride_t;
          const int w0 = (q0 + r0) >> 5;
          const int wend = (qb == p.nQ - 1 && r0 + 128 >= p.QB) ? (int)p.stride_t : min(w0 + 4, (q0 + p.QB) >> 5);
          unsigned w[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            w[c] = t_words[threadIdx.x][c];
            const int left = p.Q_LEN - (q0 + r0 + 32 * c);
            if (left < 32) w[c] &= left <= 0 ? 0u : (1u << left) - 1u;
          }
          if ((w0 & 3) == 0 && w0 + 4 <= wend) {
            *(uint4*)(dst + w0) = make_uint4(w[0], w[1], w[2], w[3]);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (w0 + c < wend) dst[w0 + c] = w[c];
          }
          for (int i = w0 + 4; i < wend; ++i) dst[i] = 0u;
        }
        __syncthreads();
      }
    }
  }
  if (p.cls == nullptr) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) s_cnt[warp] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    int c = 0;
    for (int w = 0; w < FA_SCAN_WARPS; ++w) c += s_cnt[w];
    p.cls[((long long)bh * p.nQ + qb) * p.nKV + kvb] = (signed char)(c == 0 ? 0 : (c == p.QB * p.KVB ? 2 : 1));
  }
}

// Any block size: one CTA per block counts the positions kept.
extern "C" __global__ void __launch_bounds__(256) fa_blockmask_classify_kernel(const __grid_constant__ FaMaskParams p) {
  FA_MOD_BUFS_INIT(p);
  fa_grid_wait();
  __shared__ long long s_cnt;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  const int kvb = blockIdx.x, qb = blockIdx.y;
  const int bh = blockIdx.z;
  const int b = bh / p.H, h = bh - b * p.H;
  const long long total = (long long)p.QB * p.KVB;
  int cnt = 0;
#if FA_HAS_MASK_MOD
  const int gb = b + p.b_off, gh = h + p.h_off;
  const int q0 = qb * p.QB, k0 = kvb * p.KVB;
  for (long long i = threadIdx.x; i < total; i += 256) {
    const int qi = (int)(i / p.KVB);
    const int kj = (int)(i - (long long)qi * p.KVB);
    cnt += fa_mask_mod(gb, gh, q0 + qi, k0 + kj) ? 1 : 0;
  }
#else
  for (long long i = threadIdx.x; i < total; i += 256) cnt += 1;
#endif
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if ((threadIdx.x & 31) == 0) atomicAdd((unsigned long long*)&s_cnt, (unsigned long long)cnt);
  __syncthreads();
  if (threadIdx.x == 0) {
    const long long c = s_cnt;
    p.cls[((long long)bh * p.nQ + qb) * p.nKV + kvb] = (signed char)(c == 0 ? 0 : (c == total ? 2 : 1));
  }
}
