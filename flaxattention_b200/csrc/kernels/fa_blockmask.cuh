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

// One CTA of four warps per block, in 128 x 128 sub-tiles: a warp takes 32 rows, a lane one of them, 32 keys at a time.  The
// lane's own bits over the keys are a word of the row-major matrix (one predicated OR per position), what a mask reads per
// query (a captured document id) is loaded once per lane and what it reads per key is a broadcast; five exchange steps
// between the lanes turn the 32 words into those of the transposed matrix (some 25 instructions per 1024 positions).  Both matrices and
// the block's count come out of one evaluation.  Where interval arithmetic over the mask's expression (fa_mask_range, from
// the tracer) says that 32 x 32 positions are all kept or all not, none is evaluated.  Bound by instruction issue.  8192 x 8192 positions of an attention-sink mask:
// 29 us; with lane = key, a ballot per row and a select for its word, 41.
// Needs key blocks of whole 32-bit words and query blocks of whole words or a single one; other block sizes go to the
// classify kernel below.
constexpr int FA_SCAN_WARPS = 4;
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
extern "C" __global__ void __launch_bounds__(128) fa_mask_scan_kernel(const __grid_constant__ FaMaskParams p) {
  FA_MOD_BUFS_INIT(p);
  fa_grid_wait();
  __shared__ __align__(16) unsigned t_words[128][FA_SCAN_WARPS];
  __shared__ unsigned r_words[4][128];
  __shared__ int s_cnt[FA_SCAN_WARPS];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvb = blockIdx.x, qb = blockIdx.y, bh = blockIdx.z;
  const int b = bh / p.H, h = bh - b * p.H;
  const int gb = b + p.b_off, gh = h + p.h_off;
  const int q0 = qb * p.QB, k0 = kvb * p.KVB;
  int cnt = 0;
  for (int r0 = 0; r0 < p.QB; r0 += 128) {
    const int row = r0 + warp * 32 + lane, q = q0 + row;  // this lane's row inside the block, and its query
    const bool row_in = row < p.QB;
    for (int c0 = 0; c0 < p.KVB; c0 += 128) {
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const int kv = k0 + c0 + 32 * c, left = p.KVB - (c0 + 32 * c);
        unsigned w = 0u;
        if (left > 0) {  // (the same for all threads)
          int known = 1;
#ifdef FA_HAS_MASK_RANGE
          known = fa_mask_range(gb, gh, q - lane, q - lane + 31, kv, kv + 31);  // (the same for the warp)
#endif
          if (known == 1) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (fa_mask_mod(gb, gh, q, kv + e)) w |= 1u << e;
          } else {
            w = known ? 0xffffffffu : 0u;
          }
          if (left < 32) w &= (1u << left) - 1u;
          if (!row_in) w = 0u;
        }
        cnt += __popc(w);
        r_words[c][threadIdx.x] = w;  // (read back by this thread)
        if (p.bits_t != nullptr) t_words[32 * c + lane][warp] = fa_bit_transpose(w, lane);
      }
      if (p.bits != nullptr) {
        // the row's words of this sub-tile; keys beyond KV_LEN are 0, and the last block also writes the padding words
        if (row_in && q < p.Q_LEN) {
          unsigned* dst = p.bits + ((long long)bh * p.Q_LEN + q) * p.stride;
          const int w0 = (k0 + c0) >> 5;
          const int wend = (kvb == p.nKV - 1 && c0 + 128 >= p.KVB) ? (int)p.stride : min(w0 + 4, (k0 + p.KVB) >> 5);
          unsigned roww[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int left = p.KV_LEN - (k0 + c0 + 32 * c);
            roww[c] = r_words[c][threadIdx.x];
            if (left < 32) roww[c] &= left <= 0 ? 0u : (1u << left) - 1u;
          }
          if ((w0 & 3) == 0 && w0 + 4 <= wend) {
            *(uint4*)(dst + w0) = make_uint4(roww[0], roww[1], roww[2], roww[3]);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (w0 + c < wend) dst[w0 + c] = roww[c];
          }
          for (int w = w0 + 4; w < wend; ++w) dst[w] = 0u;
        }
      }
      if (p.bits_t != nullptr) {
        __syncthreads();
        const int col = c0 + (int)threadIdx.x, kv = k0 + col;
        if (col < p.KVB && kv < p.KV_LEN) {
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
    const int c = s_cnt[0] + s_cnt[1] + s_cnt[2] + s_cnt[3];
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
