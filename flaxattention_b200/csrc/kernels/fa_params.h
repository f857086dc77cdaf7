// Kernel parameter block shared by the host library and the run-time compiled kernels.
// Only built-in types: the same text is compiled by nvcc/g++ (host) and by NVRTC (device).
#pragma once

struct FaTensor {
  void* ptr;
  long long sb, sh, ss;  // element strides of batch, head, sequence; the head dim is contiguous
};

// BlockMask tables (layout of flaxattention/core/blockmask.py:72-119): all int32.
//   kv_num [mB,mH,nQ]   kv_idx [mB,mH,nQ,nKV]   full_* same shapes or null
//   q_num  [mB,mH,nKV]  q_idx  [mB,mH,nKV,nQ]   full_* same shapes or null
// kv_num == nullptr means "no tables": one block that spans the whole key range.
struct FaTables {
  const int* kv_num;
  const int* kv_idx;
  const int* full_kv_num;
  const int* full_kv_idx;
  const int* q_num;
  const int* q_idx;
  const int* full_q_num;
  const int* full_q_idx;
  int mB, mH;    // 1 = broadcast over batch / head
  int nQ, nKV;   // number of q / kv blocks
  int QB, KVB;   // block sizes in tokens
  // optional: mask_mod evaluated once for all positions.  Bit (kv % 32) of word
  // [((bb * mask_H + hb) * mask_rows + q) * mask_stride + kv / 32] is mask_mod(b, h, q, kv), with
  // bb = b (hb = h) or 0 where the matrix is broadcast over the batch (heads).
  // Null: the kernels evaluate mask_mod themselves on partial tiles.
  const unsigned* mask_bits;
  long long mask_stride;  // words per row (a multiple of 4: rows start on 16-byte boundaries)
  int mask_rows;          // rows per (batch, head) entry
  int mask_B, mask_H;     // entries of the matrix along batch / heads (1 = broadcast)
  // the same matrix transposed, for the kernels whose threads own a key: bit (q % 32) of word
  // [((bb * mask_H + hb) * mask_t_rows + kv) * mask_t_stride + q / 32].  Null: not built.
  const unsigned* mask_bits_t;
  long long mask_t_stride;
  int mask_t_rows;
  const int* mask_hold;  // device word or null: 0 - the matrices do not hold any more, evaluate mask_mod
};

// Tensors a score_mod / mask_mod may capture and index (fa_module_set_buffers).  Their addresses travel
// with the kernel parameters; a kernel whose mods read any copies them into the table the generated code
// looks them up in (FA_MOD_BUFS_INIT), and its first block-wide barrier makes the table visible.
#define FA_MAX_MOD_BUFS 8
#ifdef FA_NUM_MOD_BUFS
#define FA_MOD_BUFS_INIT(P)                                                                      \
  do {                                                                                           \
    if (threadIdx.x < FA_NUM_MOD_BUFS) fa_mod_buf[threadIdx.x] = (P).mod_buf[threadIdx.x];       \
  } while (0)
#else
#define FA_MOD_BUFS_INIT(P) \
  do {                      \
  } while (0)
#endif

// CTAs of a (batch, head) whose decode splits are merged inside a thread-block cluster (the portable cluster size)
#define FA_DECODE_MAX_CLUSTER 8

struct FaParams {
  FaTensor q, k, v, o;
  FaTensor dout, dq, dk, dv;
  float* lse;      // [B,Hq,Sq] natural-log logsumexp (forward: output or null; backward: input)
  float* delta;    // [B,Hq,Sq] backward scratch: rowsum(O * dO)
  float* part_o;   // decode scratch [B*Hq, splits, Sq, Dv] un-normalised partial outputs
  float* part_ml;  // decode scratch [B*Hq, splits, Sq, 2] running max (log2 units) and sum
  int* status;     // optional device status word; kernels OR error bits into it
  int B, Hq, Hkv, Sq, Skv, D, Dv;
  int b_off, h_off;  // global index of this shard's first batch / head (what the mods see)
  int num_splits;
  int n_q_tiles;
  float scale;
  const void* mod_buf[FA_MAX_MOD_BUFS];
  FaTables t;
  // fp32 inputs as bf16 parts: one byte per 32 rows of q, k, v and dO, set where a value has no such parts, the
  // rows numbered through [B, H, S] (dO, backward only: S rounded up to 128)
  const unsigned char* beyond[4];
};

// Evaluation of mask_mod over a block grid: the class of every block and, optionally, the mask itself as
// bit matrices.  `B`, `H`: entries evaluated (1 where the mask does not read the batch / head index).
struct FaMaskParams {
  signed char* cls;  // [B,H,nQ,nKV]: 0 empty, 1 partial, 2 full; or null
  unsigned* bits;    // [B,H,Q_LEN,stride] words, or null
  unsigned* bits_t;  // [B,H,KV_LEN,stride_t] words, or null
  long long stride, stride_t;
  int B, H, nQ, nKV, QB, KVB, Q_LEN, KV_LEN;
  int b_off, h_off;
  const void* mod_buf[FA_MAX_MOD_BUFS];
};

#ifdef __CUDACC_RTC__
// Programmatic dependent launch: a kernel of this library may be scheduled while the one in front of it on
// the stream is finishing.  fa_grid_wait returns when that one is complete and its writes are visible
// (every kernel calls it before its first access to global memory); fa_grid_release lets the next
// kernel be scheduled as soon as every CTA of this one has called it or has exited.
__device__ __forceinline__ void fa_grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void fa_grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif
