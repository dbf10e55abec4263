// Arguments of the entry points that take structures: shared by the kernel files and by the native host module (host.cpp), mirrored
// field by field by the ctypes Structures in ops/_lib.py.
#pragma once

// Arguments of np_gemm_bf16.
struct NpGemmArgs {
  const void* A; const void* B; const void* B2; void* C; void* C2;
  long long lda, ldb, ldc, ldc2;
  long long a_rows, b_rows;  // total rows (K-major) or total K rows (MN-major) of the A / B tensors
  int M, N, K;
  // epilogue 2: C is [d gate | d up] and C2 the pre-activations [gate | up], each [M, 2 N]; the product is d h
  int a_mn, b_mn, out_f32, accumulate, epilogue, mode;
  float alpha;
  const int* mblk_group; const int* mblk_rows; long long group_stride_b;
  int num_groups, blocks_per_group; long long group_stride_c;
  const int* ready_flags; const int* mblk_flag; int epoch; unsigned long long flag_limit_ns;
  const long long* row_dst; void* const* peer_base;
  int* done_counters; const int* done_expected; int* const* done_flag_ptr;
  int bn;        // columns of a tile: 0 = choose, else 128 or 256 (128: one CTA per tile, whatever mt and split say)
  int max_ctas;  // 0 = all SMs
  const void* Cin; long long ldcin;  // optional accumulate source (defaults to C when accumulate != 0)
  const int* epoch_base;             // optional device counter added to `epoch`
  // B arriving in row shards (a sharded weight being all-gathered while the GEMM runs): the producer waits for
  // the flag of every shard a tile touches before it loads from it
  const int* b_ready_flags; int b_rows_per_flag;
  // Local shard read in place (K-major operands only): A rows [a_loc_lo, a_loc_hi) from A_loc (row 0 = a_loc_lo),
  // B rows [b_loc_lo, b_loc_hi) from B_loc; the block boundaries must be multiples of the tile size. b_local_flag:
  // 1 + index of the B flag that needs no wait (0: none). m_rot / n_rot: first M / N block of the tile order.
  const void* A_loc; long long lda_loc; int a_loc_lo, a_loc_hi;
  const void* B_loc; long long ldb_loc; int b_loc_lo, b_loc_hi;
  int b_local_flag, m_rot, n_rot;
  // all-gather pushed by the GEMM's own CTAs before their first tile: push_bytes of push_src to push_dst[r]
  // (r < push_n <= 8; the destinations already point at this rank's slot), then *push_flag[r] = epoch (+ base);
  // push_ctr: a zeroed local int
  const void* push_src; long long push_bytes; void* const* push_dst; int* const* push_flag; int push_n; int* push_ctr;
  const float* bias;  // optional [N] fp32 bias added in the plain epilogue (alpha != 0)
  // rows of a tile in units of 128: 0 = choose, 1, or 2 (256 x 256 tiles on a pair of CTAs; forms that the pair kernel does
  // not take, and launches of one CTA, run one CTA per tile)
  int mt;
  int split;          // parts of K: 0 = choose, 1, or 2 or 4 on the pair kernel (dense, plain epilogue, 8 K steps, M above 128)
  int paired;         // row-grouped form: blocks 2 i and 2 i + 1 share their group and their arrival flag
  int k_split;        // > 0 (MN-major B): K rows [0, k_split) of a group come from B, the rest from B2 (multiple of 64)
  int m_split;        // > 0: output rows [0, m_split) go to C, the rest to C2 (layout of C; multiple of 256)
  int pair_bn;        // columns of a pair's tile: 0 = choose, 128, 192 or 256
  int local_push;     // the destinations behind peer_base and done_flag_ptr are this GPU's: ordered at device scope
  int round_acc;      // epilogue 2: dh is rounded to bf16 before the gradient of the activation, as a product of its own would store it
};

// Tensor layout of q / k / v / o: [B, S, H, 128] bf16 with element strides (sb, ss, sh); the last dim is
// contiguous. k_ptrs / v_ptrs: one base pointer per KV source (n_src = 1 without context parallelism).
struct NpAttnFwdArgs {
  const void* q; long long q_sb, q_ss, q_sh;
  const void* const* k_ptrs; const void* const* v_ptrs; long long k_sb, k_ss, k_sh;
  void* o; long long o_sb, o_ss, o_sh;
  float* lse;
  int B, Sq, Hq, Hkv, causal, n_src, src_len, q_off;
  float scale;
  const int* q_blk_pos; const int* k_blk_pos;
  int split;       // unused (two softmax threads per row)
  int lse_heads;   // heads of the lse array when q / o are a head slice of larger tensors (0: Hq)
  // KV sources that peers are still pushing into this GPU's memory: flags[flag_idx[s]] >= flag_epoch + *epoch_base
  const int* src_flags; const int* flag_idx; int flag_epoch; const int* epoch_base; unsigned long long flag_limit_ns;
  int flag_own;    // 1 + flag index that guards q itself (0: none)
  // this rank's K|V shard pushed by the kernel itself: push_bytes of push_k then push_v to push_dst[r] (r < push_n),
  // then *push_flag[r] = flag_epoch (+ *epoch_base); push_ctr: two local ints the caller zeroes before the launch
  const void* push_k; const void* push_v; long long push_bytes; void* const* push_dst; int* const* push_flag;
  int push_n; int* push_ctr;
  int head_dim;    // 128 (also when 0) or 64
};

// Backward of np_attn_fwd. q / o / d_o / dq are local [B, Sq, Hq, 128]; k / v / dk / dv local
// [B, Sk, Hkv, 128]. kv sources (for dQ) and q / d_o / lse / delta sources (for dK, dV) are lists so a
// context-parallel rank reads its peers' tensors in place; without context parallelism both lists have
// one entry, the local tensors. delta = rowsum(dO o O) is computed here into `delta` ([B, Hq, Sq] fp32).
// phase: 1 = delta only, 2 = dQ + dKV only (delta already published), 3 = all.
struct NpAttnBwdArgs {
  const void* q; long long q_sb, q_ss, q_sh;
  const void* k; const void* v; long long k_sb, k_ss, k_sh;
  const void* o; long long o_sb, o_ss, o_sh;
  const void* d_o; long long do_sb, do_ss, do_sh;
  const float* lse; float* delta;
  void* dq; long long dq_sb, dq_ss, dq_sh;
  void* dk; void* dv; long long dk_sb, dk_ss, dk_sh;
  const void* const* k_src; const void* const* v_src;           // n_src KV sources (layout of k)
  const void* const* q_src; const void* const* do_src;          // n_src Q / dO sources (layouts of q / d_o)
  const float* const* lse_src; const float* const* delta_src;   // n_src [B, Hq, Sq] sources
  int B, Sq, Sk, Hq, Hkv, causal, n_src, q_off, phase;
  float scale;
  const int* q_blk_pos_local; const int* k_blk_pos_all;         // for dQ: local Q blocks vs all KV blocks
  const int* k_blk_pos_local; const int* q_blk_pos_all;         // for dKV: local KV blocks vs all Q blocks
  int split;                                                    // softmax threads per row: 2 (default) or 4
  int lse_heads;                                                // heads of the lse / delta arrays (0: Hq)
  // sources still arriving (as in NpAttnFwdArgs); which = 1: the flags guard the KV sources of the dQ kernel,
  // 2: the Q / dO / lse / delta sources of the dK/dV kernel, 3: both
  const int* src_flags; const int* flag_idx; int flag_epoch; const int* epoch_base; unsigned long long flag_limit_ns;
  int flag_which;
  int skip;       // 1: no dQ kernel, 2: no dK/dV kernel
  int flag_own;   // 1 + flag index that guards the resident operands (q, d_o, lse, delta / k, v), 0: none
  // K|V shard pushed by the dQ kernel itself (as in NpAttnFwdArgs)
  const void* push_k; const void* push_v; long long push_bytes; void* const* push_dst; int* const* push_flag;
  int push_n; int* push_ctr;
  int head_dim;    // 128 (also when 0) or 64
};

// All tensors bf16 with 16-byte aligned rows of HD elements (64 or 128).
struct NpDecodeArgs {
  const void* q; long long q_sb, q_ss, q_sh;
  const void* kc; const void* vc; long long kc_sb, kc_ss, kc_sh, vc_sb, vc_ss, vc_sh;
  const void* kn; const void* vn; long long kn_sb, kn_ss, kn_sh, vn_sb, vn_ss, vn_sh;
  void* ko; void* vo; void* o;
  int B, Sq, Hq, Hkv, past, fresh, causal, head_dim;
  float scale;
};

struct NpDispatchArgs {
  const void* x; const int* indices; const int* slot_pos; const int* counts_kept; const float* slot_scale;
  int T, K, D, E, E_local, n_ranks, my_rank, region_rows, quant;
  void* const* peer_rows; float* const* peer_scales; long long* const* peer_row_dst;
  int* const* peer_mblk_rows; int* const* peer_src_blocks; int* const* peer_flags;
  int* done_ctr; int epoch; int write_meta; int max_ctas; const int* epoch_base; int* zero_ctr;
};

struct NpCombineArgs {
  const void* rows; const int* slot_pos; const float* weights; const void* add1; const void* add2;
  const float* dl; const float* wg; void* out; int T, K, D, E;
  const int* flags; const int* sent_to_peer; int n_ranks, epoch; unsigned long long limit_ns;
  const int* epoch_base;
};

