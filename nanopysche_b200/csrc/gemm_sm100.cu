// bf16 GEMM family for sm_100a: persistent, warp-specialised, tcgen05.mma with the accumulator
// in TMEM (double buffered), operands staged by TMA into 128-byte-swizzled shared memory.
//
// One kernel covers forward (A,B K-major), dgrad (B MN-major) and wgrad (A,B MN-major), the
// ragged per-expert ("grouped") variants used by the MoE layers, a fused SwiGLU epilogue, and
// the two hooks that fuse a collective into the GEMM: a per-M-block arrival-flag wait in front
// of the loads (tokens pushed into this GPU's buffer by its peers) and an epilogue that stores
// output rows through a per-row destination table into peer memory and signals the peers.
//
// Roles per CTA (320 threads): warp 0 = TMA producer, warp 1 = MMA issuer + TMEM owner,
// warps 2..9 = epilogue (TMEM -> registers -> global). All waits are bounded (common.cuh).
//
// Replaces the cuBLAS calls behind nn.Linear / torch.bmm in the reference
// (model/attention.py:141-143,189; model/feed_forward.py:75; model/moe.py:1520-1538).
#include <cstdlib>
#include "common.cuh"
#include "args.h"

__device__ int g_np_status[8];
__device__ unsigned long long g_np_wait_end[NP_MAX_SMS];
__device__ unsigned long long g_np_wait_ns[NP_MAX_SMS];

namespace {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = 128 B = one swizzle row
constexpr int KID_GEMM = 1;

struct GemmParams {
  void* C;            // output
  void* C2;           // swiglu: optional [gate | up] pre-activation output, (M, 2*N_out)
  int M, N, K;        // output rows / cols, contraction length
  long long ldc, ldc2;
  int a_mn, b_mn;     // 0: operand is K-major ([rows, K]); 1: MN-major ([K, rows])
  int out_f32;        // 0: bf16 output, 1: fp32 output
  int accumulate;     // C += A*B (read-modify-write)
  int epilogue;       // 0 plain, 1 swiglu (B tile = 128 gate rows + 128 up rows), 2 backward of swiglu (tmC2: [gate | up])
  int mode;           // 0 dense, 1 grouped rows (per-M-block B offset), 2 grouped K (wgrad)
  float alpha;
  const int* mblk_group;      // [m blocks] group of each 128-row block (mode 1) or nullptr
  const int* mblk_rows;       // [m blocks] valid rows of each block, 0 = skip; nullptr = all
  long long group_stride_b;   // rows of B per group (mode 1)
  int num_groups;             // mode 2
  int blocks_per_group;       // mode 2: 128-row blocks of the token axis per group
  long long group_stride_c;   // mode 2: elements of C per group
  const int* ready_flags;     // arrival flags (monotone epochs) or nullptr
  const int* mblk_flag;       // [m blocks] index into ready_flags
  int epoch;
  unsigned long long flag_limit_ns;
  const long long* row_dst;   // per output row: (peer << 40) | row, or < 0 to drop; nullptr = dense
  void* const* peer_base;     // [peers] base pointer of each peer's destination buffer
  int* done_counters;         // [flags] tiles finished per destination (local)
  const int* done_expected;   // [flags] M blocks expected per destination (x n_blocks tiles each)
  int* const* done_flag_ptr;  // [flags] peer flag word to release when a destination completes
  bool local_push;            // every destination is this GPU's own memory
  bool round_acc;             // SwiGLU gradient: of dh rounded to bf16
  int parts;                  // pair kernel: K in this many parts with an accumulator each, added in the epilogue
  const void* Cin;            // accumulate source (same dtype as C), rows indexed like a dense C
  long long ldcin;
  const int* epoch_base;      // optional device counter added to `epoch` (keeps epochs valid under graph replay)
  const int* b_ready_flags;   // arrival flags of the B operand: flag i covers B rows [i * b_rows_per_flag, ...)
  int b_rows_per_flag;
  // Rows of A (K-major) / B (K-major) that this GPU produced itself are read from their source tensor through a
  // second tensor map, so nothing in this kernel waits for a copy made by another kernel of the same GPU.
  int a_loc_lo, a_loc_hi;     // A rows [lo, hi) come from tmAloc (row index - lo)
  int b_loc_lo, b_loc_hi;     // B rows [lo, hi) come from tmBloc
  int b_local_flag;           // index into b_ready_flags that needs no wait (the local shard), -1: none
  int m_rot, n_rot;           // tile order starts at this M / N block (the local shard first)
  // All-gather issued by this kernel itself: before the first tile every CTA stores its slice of `push_src` into
  // the peers' gather buffers; the CTA that finishes last releases this rank's arrival flag on every peer. The
  // grid is one resident wave, so the push never waits for a CTA that has not started.
  const uint4* push_src; long long push_vecs;
  uint4* push_dst[8]; int* push_flag[8]; int push_n;
  int* push_ctr;
  int k_split;                // > 0: B rows of K steps from here on come from tmB2 (two weights, one contraction)
  int m_split;                // > 0: output rows from here on go to C2, counted from 0 (one contraction, two outputs)
  int splits;                 // pair kernel: parts of K (cluster of 2 * splits CTAs), 1 = whole
  bool st32, st32_c2;         // rows and column chunks of C / C2 are 32-byte aligned: use 32-byte stores
  bool v16, v16_c2;           // rows of C and of the accumulate source / of C2 are 16-byte aligned: whole vectors, else elements
  bool tma_c;                 // outputs leave through shared memory and TMA stores (tmC, tmC2)
  const float* bias;          // optional [N] fp32 added to every output row (plain epilogue)
};

// 64 bytes (16 registers: 32 bf16 or 16 fp32) to a row: two 32-byte stores when the address allows it (a full sector
// per request - what a row pushed to a peer over NVLink is made of), else four 16-byte stores.
__device__ __forceinline__ void store64(void* dst, const uint32_t* o, bool st32) {
  if (st32) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(o[0]), "r"(o[1]), "r"(o[2]),
                 "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                 : "memory");
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"((char*)dst + 32), "r"(o[8]), "r"(o[9]),
                 "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15])
                 : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      reinterpret_cast<uint4*>(dst)[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
  }
}

template <class F>
__device__ __forceinline__ void for_each_k(const GemmParams& p, int g, F&& f) {
  if (p.mode != 2) {
    const int nkb = (p.K + BK - 1) / BK;
    for (int kb = 0; kb < nkb; ++kb) {
      if (!f(kb * BK)) return;
    }
  } else {
    const int b0 = g * p.blocks_per_group;
    for (int b = b0; b < b0 + p.blocks_per_group; ++b) {
      const int r = p.mblk_rows ? p.mblk_rows[b] : BM;
      if (r <= 0) continue;
      if (!f(b * BM)) return;
      if (!f(b * BM + BK)) return;
    }
  }
}

__device__ __forceinline__ int count_k(const GemmParams& p, int g) {
  if (p.mode != 2) return (p.K + BK - 1) / BK;
  int n = 0;
  const int b0 = g * p.blocks_per_group;
  for (int b = b0; b < b0 + p.blocks_per_group; ++b) {
    const int r = p.mblk_rows ? p.mblk_rows[b] : BM;
    if (r > 0) n += 2;
  }
  return n;
}

struct Tile {
  int g, m_blk, n_blk;
};

// One tile's rows are stored by this warp: publish them, count the tile against its destination and release the destination's
// flag when it is done (`need` arrivals). A system-wide fence takes some 3 us; on one GPU the device scope does.
__device__ __forceinline__ void count_done(const GemmParams& p, int fi, int need, int epoch, int lane) {
  if (p.local_push) __threadfence();
  else __threadfence_system();
  __syncwarp();
  if (lane == 0 && atomicAdd(&p.done_counters[fi], 1) + 1 == need) {
    if (p.local_push) {
      __threadfence();
      np::st_release_gpu(p.done_flag_ptr[fi], epoch);
    } else {
      __threadfence_system();
      np::st_release_sys(p.done_flag_ptr[fi], epoch);
    }
  }
}

// Operand tile in shared memory (64-wide K stage): descriptor of its first 16-wide K step, and what one K step adds to the
// (16-byte) address field. K-major: 32 bytes along the swizzled row; MN-major: 16 rows of 128 bytes.
__device__ __forceinline__ uint64_t operand_desc(uint32_t tile, int mn) {
  return np::make_smem_desc(tile, mn ? 64 * BK * 2 : 16, 1024);
}
__device__ __forceinline__ uint32_t k_step(int mn) { return mn ? 2048 >> 4 : 32 >> 4; }

// Tile order: bands of BAND M blocks, so that one wave of CTAs touches a band of A row blocks and a few B row blocks
// instead of all of A, and both operands are re-read from L2 rather than from DRAM.
__device__ __forceinline__ int fast_div(int n, int d) {   // n / d for 0 <= n < 2^24 (every role decodes every tile)
  int q = (int)((float)n * __frcp_rn((float)d));
  const int r = n - q * d;
  if (r < 0) --q;
  else if (r >= d) ++q;
  return q;
}
template <int BAND>
__device__ __forceinline__ Tile decode_tile(int t, int m_blocks, int n_blocks) {
  Tile tl;
  const int per_group = m_blocks * n_blocks;
  tl.g = t < per_group ? 0 : fast_div(t, per_group);
  const int r = t - tl.g * per_group;
  const int first_m = fast_div(r, BAND * n_blocks) * BAND;
  const int gsize = (m_blocks - first_m) < BAND ? (m_blocks - first_m) : BAND;
  const int within = r - first_m * n_blocks;
  tl.n_blk = gsize == BAND ? within / BAND : fast_div(within, gsize);
  tl.m_blk = first_m + within - tl.n_blk * gsize;
  return tl;
}

// Where a thread's output row goes. Row-table launches: into the peer named by the table; rows and columns outside the
// output are not stored.
struct OutRow {
  char* c;
  const char* cin;   // accumulate source or nullptr
  bool ok;
};
__device__ __forceinline__ OutRow out_row(const GemmParams& p, int g, int row) {
  OutRow o;
  const int es = p.out_f32 ? 4 : 2;
  o.ok = row < p.M;
  if (p.m_split && row >= p.m_split) {
    o.c = (char*)p.C2 + ((size_t)g * p.group_stride_c + (size_t)(row - p.m_split) * p.ldc) * es;
    o.cin = p.Cin ? o.c : nullptr;       // the accumulating form adds to its own output
    return o;
  }
  if (p.row_dst) {
    const long long d = o.ok ? p.row_dst[row] : -1;
    o.ok = o.ok && d >= 0;
    const long long peer = o.ok ? (d >> 40) : 0;
    const long long drow = d & ((1ll << 40) - 1);
    o.c = (char*)p.peer_base[peer] + (size_t)drow * p.ldc * es;
  } else {
    o.c = (char*)p.C + ((size_t)g * p.group_stride_c + (size_t)row * p.ldc) * es;
  }
  o.cin = p.Cin ? (const char*)p.Cin + ((size_t)g * p.group_stride_c + (size_t)row * p.ldcin) * es : nullptr;
  return o;
}

// 32 accumulator columns from output column `col`: times alpha, plus bias. The conditions are outside the loops: tested per
// element they cost more than the rest of the epilogue.
__device__ __forceinline__ void scale_bias(const GemmParams& p, uint32_t* r, int col) {
  if (p.alpha != 1.f) {
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * p.alpha);
  }
  if (p.bias) {   // the same 32 values for every row of the warp: broadcast loads
    if (col + 32 <= p.N) {
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + p.bias[col + i]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (col + i < p.N) r[i] = __float_as_uint(__uint_as_float(r[i]) + p.bias[col + i]);
    }
  }
}
__device__ __forceinline__ void pack32(const uint32_t* r, uint32_t* w) {
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = np::pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}

// Plain epilogue of 32 accumulator columns, stored from the registers (accumulate sources, peer rows, odd alignments).
__device__ __forceinline__ void store_chunk(const GemmParams& p, const OutRow& o, uint32_t* r, int col) {
  if (!o.ok || col >= p.N) return;
  scale_bias(p, r, col);
  if (p.v16 && col + 32 <= p.N) {
    if (o.cin) {
      if (p.out_f32) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 c = reinterpret_cast<const float4*>((const float*)o.cin + col)[i];
          r[4 * i] = __float_as_uint(__uint_as_float(r[4 * i]) + c.x);
          r[4 * i + 1] = __float_as_uint(__uint_as_float(r[4 * i + 1]) + c.y);
          r[4 * i + 2] = __float_as_uint(__uint_as_float(r[4 * i + 2]) + c.z);
          r[4 * i + 3] = __float_as_uint(__uint_as_float(r[4 * i + 3]) + c.w);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 c = reinterpret_cast<const uint4*>((const __nv_bfloat16*)o.cin + col)[i];
          const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 f = np::unpack_bf16(cw[q]);
            r[8 * i + 2 * q] = __float_as_uint(__uint_as_float(r[8 * i + 2 * q]) + f.x);
            r[8 * i + 2 * q + 1] = __float_as_uint(__uint_as_float(r[8 * i + 2 * q + 1]) + f.y);
          }
        }
      }
    }
    if (p.out_f32) {
      float* dst = (float*)o.c + col;
      store64(dst, r, p.st32);
      store64(dst + 16, r + 16, p.st32);
    } else {
      uint32_t w[16];
      pack32(r, w);
      store64((__nv_bfloat16*)o.c + col, w, p.st32);
    }
    return;
  }
  _Pragma("unroll") for (int i = 0; i < 32; ++i) if (col + i < p.N) {
    float v = __uint_as_float(r[i]);
    if (p.out_f32) {
      if (o.cin) v += ((const float*)o.cin)[col + i];
      ((float*)o.c)[col + i] = v;
    } else {
      if (o.cin) v += __bfloat162float(((const __nv_bfloat16*)o.cin)[col + i]);
      ((__nv_bfloat16*)o.c)[col + i] = __float2bfloat16(v);
    }
  }
}

// SwiGLU epilogue of 32 gate and 32 up columns: silu(gate) * up, and the pre-activations side by side when asked for.
__device__ __forceinline__ void store_swiglu_chunk(const GemmParams& p, const OutRow& o, const uint32_t* g, const uint32_t* u,
                                                   int row, int col) {
  if (!o.ok || col >= p.N) return;
  const bool full = col + 32 <= p.N;
  uint32_t h[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float g0 = __uint_as_float(g[2 * i]), g1 = __uint_as_float(g[2 * i + 1]);
    const float u0 = __uint_as_float(u[2 * i]), u1 = __uint_as_float(u[2 * i + 1]);
    h[i] = np::pack_bf16(np::silu_f(g0) * u0, np::silu_f(g1) * u1);
  }
  __nv_bfloat16* dst = (__nv_bfloat16*)o.c + col;
  if (full && p.v16) {
    store64(dst, h, p.st32);
  } else {
    _Pragma("unroll") for (int i = 0; i < 32; ++i) if (col + i < p.N) dst[i] = reinterpret_cast<__nv_bfloat16*>(h)[i];
  }
  if (!p.C2) return;
  __nv_bfloat16* d2 = (__nv_bfloat16*)p.C2 + (size_t)row * p.ldc2 + col;
  if (full && p.v16_c2) {
#pragma unroll
    for (int i = 0; i < 16; ++i) h[i] = np::pack_bf16(__uint_as_float(g[2 * i]), __uint_as_float(g[2 * i + 1]));
    store64(d2, h, p.st32_c2);
#pragma unroll
    for (int i = 0; i < 16; ++i) h[i] = np::pack_bf16(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1]));
    store64(d2 + p.N, h, p.st32_c2);
  } else {
    _Pragma("unroll") for (int i = 0; i < 32; ++i) if (col + i < p.N) {
      d2[i] = __float2bfloat16(__uint_as_float(g[i]));
      d2[p.N + i] = __float2bfloat16(__uint_as_float(u[i]));
    }
  }
}

// Two warps share the 32 tensor-memory lanes of a quarter and take half of a tile's columns each: the drain of a tile
// that no MMA of a next tile covers (the only, or the last one of a CTA) takes half as long as with one.
constexpr int EPI_WARPS = 8;
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
constexpr int STG_BYTES = 4096;   // staging of one epilogue warp: 32 rows of 128 bytes

// A warp's 32 rows of 128 bytes (w: this lane's row, 32 words) to the output at (col, row0, plane): through the warp's
// staging buffer, in the 128-byte swizzle of the tensor map, and one TMA store. Stored straight from the registers every
// instruction touches 32 rows, one sector each: a 128 x 256 fp32 tile took about 10 us that way.
__device__ __forceinline__ void stage_store(const CUtensorMap* tm, uint32_t stg, int lane, const uint32_t* w, int col, int row0,
                                            int plane) {
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the buffer's last store has read it
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stg + lane * 128 + ((j ^ (lane & 7)) << 4)), "r"(w[4 * j]),
                 "r"(w[4 * j + 1]), "r"(w[4 * j + 2]), "r"(w[4 * j + 3])
                 : "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(tm), "r"(stg), "r"(col),
                 "r"(row0), "r"(plane)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}
// Backward of h = silu(gate) * up, 32 columns of dh at a time: the pre-activations of the same rows and columns arrive by TMA
// in the warp's staging buffer (gate box, up box: 32 rows of 64 bytes each, 64-byte swizzle), d(gate) and d(up) are written
// over them and leave the same way. dh itself never reaches memory: as a pass of its own this was 46 us of a 720 us
// feed-forward (4096 tokens, 2048 x 5632), 92 MB of it dh written and read.
struct GluBar {   // of one epilogue warp, over all its tiles
  uint32_t bar, phase;
};
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(tm), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
template <int BN>
__device__ __forceinline__ void store_glu_bwd(const GemmParams& p, const CUtensorMap* tmD, const CUtensorMap* tmGU, uint32_t stg,
                                              GluBar& gb, volatile int* abort_flag, uint32_t taddr, int row0, int lane, int n0,
                                              int half) {
  if (row0 >= p.M) return;
#pragma unroll 1
  for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
    const int col = n0 + c * 32;
    if (col >= p.N) break;
    if (lane == 0) {
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the last boxes have left
      np::mbar_expect_tx(gb.bar, 4096);
      tma_load_3d(stg, tmGU, gb.bar, col, row0, 0);
      tma_load_3d(stg + 2048, tmGU, gb.bar, col, row0, 1);
    }
    __syncwarp();
    uint32_t r[32];
    np::tmem_ld32(taddr + c * 32, r);
    np::tmem_ld_wait();
    if (!np::mbar_wait_warp(gb.bar, gb.phase, abort_flag, KID_GEMM, 16)) return;
    gb.phase ^= 1u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {   // 8 columns: 16 bytes of gate and of up
      const uint32_t at = stg + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4);
      uint32_t g[4], u[4], dg[4], du[4];
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(g[0]), "=r"(g[1]), "=r"(g[2]), "=r"(g[3]) : "r"(at) : "memory");
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(at + 2048) : "memory");
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 gf = np::unpack_bf16(g[q]), uf = np::unpack_bf16(u[q]);
        float d0 = __uint_as_float(r[8 * j + 2 * q]) * p.alpha, d1 = __uint_as_float(r[8 * j + 2 * q + 1]) * p.alpha;
        if (p.round_acc) {
          const float2 d = np::unpack_bf16(np::pack_bf16(d0, d1));
          d0 = d.x;
          d1 = d.y;
        }
        const float s0 = np::sigmoid_f(gf.x), s1 = np::sigmoid_f(gf.y);
        dg[q] = np::pack_bf16(d0 * uf.x * (s0 * (1.f + gf.x * (1.f - s0))), d1 * uf.y * (s1 * (1.f + gf.y * (1.f - s1))));
        du[q] = np::pack_bf16(d0 * (gf.x * s0), d1 * (gf.y * s1));
      }
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(dg[0]), "r"(dg[1]), "r"(dg[2]), "r"(dg[3]) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 2048), "r"(du[0]), "r"(du[1]), "r"(du[2]), "r"(du[3]) : "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
#pragma unroll
      for (int z = 0; z < 2; ++z)
        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(tmD),
                     "r"(stg + z * 2048), "r"(col), "r"(row0), "r"(z)
                     : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
}

// Before the CTA exits: the staging buffer has been read.
__device__ __forceinline__ void stage_drain(int lane) {
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// 32 accumulator columns of this lane's row (zeros without an accumulator)
__device__ __forceinline__ void load_acc(uint32_t taddr, bool have_acc, uint32_t* r) {
  if (have_acc) {
    np::tmem_ld32(taddr, r);
    np::tmem_ld_wait();
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = 0u;
  }
}

// Half `half` of the BN accumulator columns of one 128-row tile: tensor memory (`taddr`: this warp's lanes, first column)
// through the epilogue of the launch to output rows row0 .. row0 + 31, columns from `n0`. Executed by whole warps (the
// tensor-memory loads are .sync.aligned).
template <int BN>
__device__ __forceinline__ void store_tile(const GemmParams& p, const CUtensorMap* tmC, const CUtensorMap* tmC2, uint32_t stg,
                                           uint32_t taddr, int g_idx, int row0, int lane, int n0, int half, bool have_acc) {
  if (p.tma_c) {
    if (row0 >= p.M) return;
    if (p.m_split && row0 >= p.m_split) {
      tmC = tmC2;
      row0 -= p.m_split;
    }
    if (p.epilogue == 1) {
      // BN / 2 output columns: 64 per warp for BN = 256; h, then the gate and the up pre-activations
#pragma unroll 1
      for (int c = half * (BN / 256); c < (half + 1) * (BN / 256); ++c) {
        const int col = n0 + c * 64;
        if (col >= p.N) break;
        uint32_t w[32];
#pragma unroll 1
        for (int out = 0; out < (p.C2 ? 3 : 1); ++out) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t g[32], u[32];
            const uint32_t tg = taddr + c * 64 + q * 32;
            if (out == 0) {
              np::tmem_ld32(tg, g);
              np::tmem_ld32(tg + BN / 2, u);
              np::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i)
                g[i] = __float_as_uint(np::silu_f(__uint_as_float(g[i])) * __uint_as_float(u[i]));
            } else {
              np::tmem_ld32(out == 1 ? tg : tg + BN / 2, g);
              np::tmem_ld_wait();
            }
            pack32(g, w + 16 * q);
          }
          stage_store(out == 0 ? tmC : tmC2, stg, lane, w, col, row0, out == 2 ? 1 : 0);
        }
      }
    } else if (p.out_f32) {
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        const int col = n0 + c * 32;
        if (col >= p.N) break;
        uint32_t r[32];
        load_acc(taddr + c * 32, have_acc, r);
        scale_bias(p, r, col);
        stage_store(tmC, stg, lane, r, col, row0, g_idx);
      }
    } else {
#pragma unroll 1
      for (int c = half; c < BN / 64; c += 2) {   // 192 columns: two chunks for one warp of a quarter, one for the other
        const int col = n0 + c * 64;
        if (col >= p.N) break;
        uint32_t w[32];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t r[32];
          load_acc(taddr + c * 64 + q * 32, have_acc, r);
          scale_bias(p, r, col + q * 32);
          pack32(r, w + 16 * q);
        }
        stage_store(tmC, stg, lane, w, col, row0, g_idx);
      }
    }
    return;
  }
  const int row = row0 + lane;
  const OutRow o = out_row(p, g_idx, row);
  if (p.epilogue == 1) {
    // gate = columns [0, BN/2), up = columns [BN/2, BN)
#pragma unroll 1
    for (int c = half * (BN / 128); c < (half + 1) * (BN / 128); ++c) {
      uint32_t g[32], u[32];
      __syncwarp();   // rows that are not stored leave the chunk early
      np::tmem_ld32(taddr + c * 32, g);
      np::tmem_ld32(taddr + BN / 2 + c * 32, u);
      np::tmem_ld_wait();
      store_swiglu_chunk(p, o, g, u, row, n0 + c * 32);
    }
  } else {
#pragma unroll 1
    for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
      uint32_t r[32];
      __syncwarp();
      load_acc(taddr + c * 32, have_acc, r);
      store_chunk(p, o, r, n0 + c * 32);
    }
  }
}

// One CTA per tile: a 128 x BN accumulator, double-buffered in tensor memory (the epilogue of a tile runs under the
// MMAs of the next).
template <int BN, int STAGES>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmAloc,
                 const __grid_constant__ CUtensorMap tmBloc, const __grid_constant__ CUtensorMap tmC,
                 const __grid_constant__ CUtensorMap tmC2, const GemmParams p) {
  constexpr int A_BYTES = BM * BK * 2;
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = (2 * BN <= 32) ? 32 : (2 * BN <= 64 ? 64 : (2 * BN <= 128 ? 128 : (2 * BN <= 256 ? 256 : 512)));

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (np::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t stg_base = smem_base + STAGES * STAGE_BYTES;   // staging of the epilogue warps
  const uint32_t bar_base = stg_base + EPI_WARPS * STG_BYTES;
  // barriers: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]; then tmem ptr, abort flag
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  uint8_t* tail = smem_raw + (bar_base - np::smem_u32(smem_raw)) + 8 * (2 * STAGES + 4 + EPI_WARPS);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  const int m_blocks = (p.M + BM - 1) / BM;
  const int bn_out = (p.epilogue == 1) ? BN / 2 : BN;  // output columns per tile
  const int n_blocks = (p.N + bn_out - 1) / bn_out;
  const int groups = (p.mode == 2) ? p.num_groups : 1;
  const int tiles_per_group = m_blocks * n_blocks;
  const int num_tiles = tiles_per_group * groups;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      np::mbar_init(full_bar(s), 1);
      np::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      np::mbar_init(tfull_bar(a), 1);
      np::mbar_init(tempty_bar(a), EPI_WARPS);
    }
    for (int w = 0; w < EPI_WARPS; ++w) np::mbar_init(bar_base + 8u * (2 * STAGES + 4 + w), 1);
    *abort_flag = 0;
    np::mbar_fence_init();
  }
  if (threadIdx.x == 64) {   // while another warp sets up the barriers
    np::tma_prefetch_desc(&tmA);
    np::tma_prefetch_desc(&tmB);
    if (p.tma_c) np::tma_prefetch_desc(&tmC);
    if (p.tma_c && p.C2) np::tma_prefetch_desc(&tmC2);
  }
  if (warp == 1) {
    np::tmem_alloc(np::smem_u32((const void*)tmem_ptr_smem), TMEM_COLS);
    np::tmem_relinquish();
  }
  np::tc_fence_before();
  __syncthreads();
  np::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  np::pdl_begin();
  const int epoch = p.epoch + (p.epoch_base ? *p.epoch_base : 0);

  if (p.push_src) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.push_vecs;
         i += (long long)gridDim.x * blockDim.x) {
      const uint4 v = p.push_src[i];
      for (int r = 0; r < p.push_n; ++r) p.push_dst[r][i] = v;
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(p.push_ctr, 1) == (int)gridDim.x - 1) {
      __threadfence_system();
      for (int r = 0; r < p.push_n; ++r) np::st_release_sys(p.push_flag[r], epoch);
      *p.push_ctr = 0;
    }
  }

  auto decode = [&](int t) {
    Tile tl = decode_tile<16>(t, m_blocks, n_blocks);
    if (p.m_rot) tl.m_blk = (tl.m_blk + p.m_rot) % m_blocks;
    if (p.n_rot) tl.n_blk = (tl.n_blk + p.n_rot) % n_blocks;
    return tl;
  };
  // rows of this M block that carry data (0 = nothing to do); waits for the arrival flag first.
  auto tile_rows = [&](const Tile& tl, int role) -> int {
    if (p.mode != 1) return BM;
    if (p.ready_flags) {
      const int fi = p.mblk_flag ? p.mblk_flag[tl.m_blk] : 0;
      if (fi >= 0 && !np::wait_flag_ge(p.ready_flags + fi, epoch, p.flag_limit_ns, KID_GEMM, 100 + role)) {
        *abort_flag = 1;
        return -1;
      }
    }
    return p.mblk_rows ? p.mblk_rows[tl.m_blk] : BM;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    // The whole warp runs the loop and elects the lane that issues, as the MMA warp does: issued by one lane of a divergent
    // branch, the loads of a K step took 230 ns whatever their size (24 to 32 KB, 4 to 128 CTAs), more than its MMAs.
    int stage = 0;
    uint32_t phase = 0;
    bool live = true;
    for (int t = blockIdx.x; t < num_tiles && live; t += gridDim.x) {
      const Tile tl = decode(t);
      const int rows = __shfl_sync(0xffffffffu, lane == 0 ? tile_rows(tl, 0) : 0, 0);
      if (rows < 0) break;
      if (rows == 0) continue;
      const int m0 = tl.m_blk * BM;
      const int n0 = tl.n_blk * bn_out;
      long long goff = 0;  // row offset of this tile's group inside the stacked B tensor
      if (p.mode == 1 && p.mblk_group) goff = (long long)p.mblk_group[tl.m_blk] * p.group_stride_b;
      const long long brow = n0 + (p.b_mn ? 0 : goff);
      const int bk_off = p.b_mn ? (int)goff : 0;
      int b_flag_hi = -1;   // highest B shard this tile has already waited for (its row ranges only move up)
      auto wait_b_rows = [&](long long r0, long long r1) -> bool {   // rows [r0, r1] of B are about to be loaded
        if (!p.b_ready_flags) return true;
        bool ok = true;
        if (lane == 0) {
          const int f0 = (int)(r0 / p.b_rows_per_flag), f1 = (int)(r1 / p.b_rows_per_flag);
          for (int f = f0 > b_flag_hi ? f0 : b_flag_hi + 1; f <= f1 && ok; ++f)
            if (f != p.b_local_flag) ok = np::wait_flag_ge(p.b_ready_flags + f, epoch, p.flag_limit_ns, KID_GEMM, 110);
          if (!ok) *abort_flag = 1;
          if (f1 > b_flag_hi) b_flag_hi = f1;
        }
        live = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        return live;
      };
      if (!p.b_mn) {
        const long long last = brow + bn_out - 1 < p.N + goff - 1 ? brow + bn_out - 1 : p.N + goff - 1;
        if (!wait_b_rows(brow, last)) break;
      }
      const bool a_loc = m0 >= p.a_loc_lo && m0 < p.a_loc_hi, b_loc = brow >= p.b_loc_lo && brow < p.b_loc_hi;
      for_each_k(p, tl.g, [&](int k0) -> bool {
        if (p.b_mn && p.b_ready_flags) {
          const long long last = k0 + bk_off + BK - 1 < p.K + bk_off - 1 ? k0 + bk_off + BK - 1 : p.K + bk_off - 1;
          if (!wait_b_rows(k0 + bk_off, last)) return false;
        }
        live = np::mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag, KID_GEMM, 1);
        if (!live) return false;
        if (np::elect_one()) {
          const uint32_t sA = smem_base + stage * STAGE_BYTES;
          const uint32_t sB = sA + A_BYTES;
          np::mbar_expect_tx(full_bar(stage), STAGE_BYTES);
          if (!p.a_mn) {
            if (a_loc) np::tma_load_2d(sA, &tmAloc, full_bar(stage), k0, m0 - p.a_loc_lo);
            else np::tma_load_2d(sA, &tmA, full_bar(stage), k0, m0);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c)
              np::tma_load_2d(sA + c * (64 * BK * 2), &tmA, full_bar(stage), m0 + c * 64, k0);
          }
          if (!p.b_mn) {
            if (p.epilogue == 1) {
              np::tma_load_2d(sB, &tmB, full_bar(stage), k0, (int)brow);
              np::tma_load_2d(sB + (BN / 2) * BK * 2, &tmB2, full_bar(stage), k0, (int)brow);
            } else if (b_loc) {
              np::tma_load_2d(sB, &tmBloc, full_bar(stage), k0, (int)brow - p.b_loc_lo);
            } else {
              np::tma_load_2d(sB, &tmB, full_bar(stage), k0, (int)brow);
            }
          } else {
            const bool second = p.k_split && k0 >= p.k_split;
            const CUtensorMap* bm = second ? &tmB2 : &tmB;
            const int kb = k0 + bk_off - (second ? p.k_split : 0);
#pragma unroll
            for (int c = 0; c < BN / 64; ++c)
              np::tma_load_2d(sB + c * (64 * BK * 2), bm, full_bar(stage), (int)brow + c * 64, kb);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        return true;
      });
    }
    if (*abort_flag) __nanosleep(1000000);  // let copies already issued land before exit
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = np::make_idesc(BM, BN, 1, 1, p.a_mn, p.b_mn);
    const uint64_t a_desc0 = operand_desc(smem_base, p.a_mn), b_desc0 = operand_desc(smem_base + A_BYTES, p.b_mn);
    const uint32_t a_step = k_step(p.a_mn), b_step = k_step(p.b_mn);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const Tile tl = decode(t);
      const int rows = __shfl_sync(0xffffffffu, lane == 0 ? tile_rows(tl, 1) : 0, 0);
      if (rows < 0) break;
      if (rows == 0) continue;
      if (count_k(p, tl.g) == 0) continue;
      if (!np::mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag, KID_GEMM, 2)) break;
      np::tc_fence_after();
      const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
      uint32_t accum = 0;
      for_each_k(p, tl.g, [&](int) -> bool {
        if (!np::mbar_wait_warp(full_bar(stage), phase, abort_flag, KID_GEMM, 3)) return false;
        np::tc_fence_after();
        if (np::elect_one()) {
          const uint64_t ad = a_desc0 + (uint32_t)(stage * (STAGE_BYTES >> 4)), bd = b_desc0 + (uint32_t)(stage * (STAGE_BYTES >> 4));
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            np::tc_mma_f16(tmem_d, ad + kk * a_step, bd + kk * b_step, idesc, kk ? 1u : accum);
          np::tc_commit(empty_bar(stage));  // frees the stage once these MMAs have read it
        }
        __syncwarp();
        accum = 1;
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        return true;
      });
      if (np::elect_one()) np::tc_commit(tfull_bar(acc));
      __syncwarp();
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
    if (*abort_flag) __nanosleep(1000000);
  } else {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3, half = (warp - 2) >> 2;  // TMEM lanes [32*quarter, 32*quarter+32), column half
    GluBar gb{bar_base + 8u * (2 * STAGES + 4 + warp - 2), 0u};
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles && !*abort_flag; t += gridDim.x) {
      const Tile tl = decode(t);
      const int rows = tile_rows(tl, 2);
      if (rows < 0) break;
      if (rows == 0) continue;
      const int nk = count_k(p, tl.g);
      const int n0 = tl.n_blk * bn_out;
      bool have_acc = nk > 0;
      if (have_acc) {
        if (!np::mbar_wait(tfull_bar(acc), acc_phase, abort_flag, KID_GEMM, 4)) break;
        np::tc_fence_after();
      }
      const uint32_t taddr = tmem_base + (uint32_t)(acc * BN) + ((uint32_t)(quarter * 32) << 16);
      const uint32_t stg = stg_base + (warp - 2) * STG_BYTES;
      const int row0 = tl.m_blk * BM + quarter * 32;
      if (p.epilogue == 2) store_glu_bwd<BN>(p, &tmC, &tmC2, stg, gb, abort_flag, taddr, row0, lane, n0, half);
      else store_tile<BN>(p, &tmC, &tmC2, stg, taddr, tl.g, row0, lane, n0, half, have_acc);
      if (have_acc) {
        np::tc_fence_before();
        __syncwarp();
        if (lane == 0) np::mbar_arrive(tempty_bar(acc));
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
      if (p.done_counters) {   // each epilogue warp counts once per tile; done_expected counts M blocks
        const int fi = p.mblk_flag ? p.mblk_flag[tl.m_blk] : 0;
        count_done(p, fi, EPI_WARPS * n_blocks * p.done_expected[fi], epoch, lane);
      }
    }
    if (p.tma_c) stage_drain(lane);
  }

  np::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    np::tc_fence_after();
    np::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------- two CTAs per tile
// A 256 x 256 tile computed by a cluster of two CTAs (tcgen05 cta_group::2): each CTA stages 128 rows of A and 128 of
// the 256 rows of B, the leader issues one 256 x 256 x 16 MMA that reads both CTAs' shared memory, and each CTA's tensor
// memory receives its own 128 rows of the result. Against the one-CTA 128 x 256 tile, which asks the L2 -> SM fabric for
// 48 KB per 64-wide K step and SM, this needs 32 KB for the same FLOPs, and unlike a 256 x 256 tile on one SM the
// 128 x 256 accumulator still fits tensor memory twice, so a tile drains under the MMAs of the next. The freed shared
// memory deepens the pipeline to six K steps (eight of 128 columns). No load is multicast.
//
// Barriers: full[s] lives in the leader and counts the bytes of both CTAs' loads; empty[s] and tfull[a] exist in both
// CTAs and are signalled by one multicast commit of the leader; tempty[a] lives in the leader and takes the arrivals of
// the epilogue warps of both CTAs. The cluster barrier at the end keeps a CTA's shared memory alive until its peer's last
// remote arrival; both CTAs reach it on every path because every wait before it is bounded.
//
// Tiles of 256 x 192 and 256 x 128 run the same way, for outputs that 256 x 256 tiles leave SMs without work on or whose last
// wave they leave nearly empty (us, 256 / 192 / 128 columns: 2048 x 3072 x 1024 16.2 / 14.9 / 17.1, 2331 x 2048 x 2048 25.2 /
// 21.4 / 26.1, 2048 x 1024 x 2816 19.0 / 16.5 / 15.3).
template <int BN>
constexpr int pair_stages() { return BN == 128 ? 8 : 6; }
// per CTA: its rows of A and half of the rows of B, in whole 64-column chunks when B is MN-major
template <int BN>
constexpr int pair_stage_bytes() { return BM * BK * 2 + (BN / 2 + 63) / 64 * 64 * BK * 2; }

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t smem_addr, uint32_t cta) {   // the same offset in another CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// load into this CTA's shared memory, bytes counted on a barrier of either CTA of the pair (not a multicast)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(tm), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair whose leader has cluster rank `leader`
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint32_t leader) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)(3u << leader))
      : "memory");
}

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, const uint32_t* v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}

// SPLIT: a cluster of `splits` pairs computes one tile, each pair a contiguous part of the K steps. When all of them are
// done, the operand stages are free: every pair sends the others their share of the columns (256 / splits each, fp32,
// through distributed shared memory), sums its own share in the order of the parts and runs the epilogue on it. No
// workspace, no atomics, and the same result every time. It is for outputs with too few tiles to occupy the SMs: the time
// of such a GEMM is its K steps one after the other (about 0.3 us each), not its FLOPs.
//
// p.parts: one pair forms the same parts in turn, each in accumulator columns of its own (128-column tiles: two parts in each of the
// two buffers; wider ones: one), and the epilogue warps add them in their order, so that the result has the bits of the cluster's. It
// takes a tile as long as a whole sum and a little more: us, whole / two parts / four / cluster of two / of four, 2048 x 1024 x 3072 17.2 /
// 17.4 / 17.9 / 17.6 / 42.6, 1024 x 768 x 2048 11.7 / 12.0 / 12.4 / 14.0 / 13.9, 768 x 768 x 4096 20.4 / 20.7 / 21.1 / 19.1 / 16.8. Tiles of 192 and
// 256 columns sum in parts beside another product only: alone, no products cover their drain (2048 x 1024 x 3072 18.7 and 20.9).
//
// DUAL: two products in one launch. A backward pass asks for the gradients of a layer's input and of its weight at the same
// time; alone, each leaves SMs without work in its only or last wave and pays for a launch, first loads and a last drain of its
// own. A pair takes its tiles of the product with the longer contraction first, then those of the other. us, two launches /
// one, in a graph, gradients of a layer of T tokens, N outputs, K inputs: T N K = 2048 1024 1024 23.2 / 14.9, 2048 3072 1024 34.8 /
// 28.4, 2048 5632 1024 50.8 / 39.3, 2331 2048 2048 43.6 / 29.8, 4096 2048 5632 with the SwiGLU gradient 178.7 / 155.9.
struct PairMaps {
  CUtensorMap A, B, B2, C, C2;
};
struct PairSecond {
  PairMaps m;
  GemmParams p;
  int extra;   // tiles of the second product that a pair with one tile less of the first takes before the rest is dealt to all
};
struct PairWork {
  int which, t;   // product and its tile; t < 0: no more
};
// Piece k of a pair's work: n0 tiles of the first product dealt in turn, then n1 of the second. Where the first do not come
// out even, the pairs from r on have one less and take up to `extra` of the second each; the rest goes to all, those pairs first.
__host__ __device__ __forceinline__ PairWork pair_work(int k, int pair, int pairs, int n0, int n1, int extra) {
  const int own = n0 > pair ? (n0 - pair - 1) / pairs + 1 : 0;
  if (k < own) return {0, pair + k * pairs};
  k -= own;
  const int r = n0 % pairs;
  int base = 0;
  if (r > 0) {
    const int slack = pairs - r;
    if (pair >= r) {
      if (k < extra) {
        const int j = pair - r + k * slack;
        return {1, j < n1 ? j : -1};
      }
      k -= extra;
    }
    base = extra < (n1 + slack - 1) / slack ? extra * slack : n1;
  }
  const int j = base + (pair >= r ? pair - r : pair - r + pairs) + k * pairs;
  return {1, j < n1 ? j : -1};
}

// K in parts: PER_BUFFER of them side by side in one of the two accumulator buffers, the rest likewise in the other
template <int BN>
constexpr int PER_BUFFER = BN == 128 ? 2 : 1;
// The parts of a tile added in their order, in place of the first (`t`: this warp's lanes, first column; `t2`: the other buffer). A pass of
// its own before the epilogue, which then is that of a whole sum: added as each epilogue form reads its columns, the parts took a captured
// step of four 350m layers from 2320 to 2404 us (launches without parts too: code that has to be fetched), with a kernel of their own
// beside the one for whole sums 2420, like this 2358. A warp adds the columns that it stores: `wide`, every other 64 of them
// (store_tile), else a half.
template <int BN>
__device__ __forceinline__ void add_parts(uint32_t t, uint32_t t2, int parts, int half, bool wide) {
#pragma unroll 1
  for (int c = 0; c < BN / 32; ++c) {
    if ((wide ? c >> 1 & 1 : c / (BN / 64)) != half) continue;
    uint32_t sum[32], v[32];
    np::tmem_ld32(t + c * 32, sum);
#pragma unroll 1
    for (int p = 1; p < parts; ++p) {
      np::tmem_ld32((p / PER_BUFFER<BN> ? t2 : t) + p % PER_BUFFER<BN> * BN + c * 32, v);
      np::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) sum[i] = __float_as_uint(__uint_as_float(sum[i]) + __uint_as_float(v[i]));
    }
    np::tmem_st16(t + c * 32, sum);
    np::tmem_st16(t + c * 32 + 16, sum + 16);
  }
  np::tmem_st_wait();
}

template <bool SPLIT, int BN, bool DUAL>
__device__ __forceinline__ void pair_body(const PairMaps& maps, const GemmParams& p, const PairSecond* second) {
  constexpr int STAGES = pair_stages<BN>(), TM = 2 * BM, HN = BN / 2;
  constexpr int A_BYTES = BM * BK * 2, STAGE_BYTES = pair_stage_bytes<BN>();
  static_assert(!SPLIT || BN == 256, "K in parts over a cluster: 256 columns");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (np::smem_u32(smem_raw) + 1023u) & ~1023u;   // the same offset in both CTAs
  const uint32_t stg_base = smem_base + STAGES * STAGE_BYTES;   // staging of the epilogue warps
  const uint32_t bar_base = stg_base + EPI_WARPS * STG_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  uint8_t* tail = smem_raw + (bar_base - np::smem_u32(smem_raw)) + 8 * (2 * STAGES + 4 + EPI_WARPS);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank(), lead = crank & ~1u;
  const int rank = (int)(crank & 1u);                              // 0: leader of its pair
  const int splits = SPLIT ? p.splits : 1, split = SPLIT ? (int)(crank >> 1) : 0;
  const int pair = (int)blockIdx.x / (2 * splits), pairs = (int)gridDim.x / (2 * splits);
  const int bn_out = (!DUAL && p.epilogue == 1) ? HN : BN;
  auto m_blocks = [&](const GemmParams& q) { return (q.M + TM - 1) / TM; };
  auto n_blocks = [&](const GemmParams& q) { return (q.N + bn_out - 1) / bn_out; };
  auto num_tiles = [&](const GemmParams& q) { return m_blocks(q) * n_blocks(q) * ((q.mode == 2) ? q.num_groups : 1); };
  const int tiles0 = num_tiles(p), tiles1 = DUAL ? num_tiles(second->p) : 0;
  // parts that this pair sums one after the other, and columns of one of the two accumulator buffers. A product alone is summed in parts
  // on 128 columns only: code that is not there does not have to be fetched
  constexpr bool PARTS = DUAL || BN == 128;
  auto k_parts = [](const GemmParams& q) { return PARTS ? q.parts : 1; };
  const int acc_cols = k_parts(p) > 1 || (DUAL && k_parts(second->p) > 1) ? PER_BUFFER<BN> * BN : BN;
  const uint32_t tmem_cols = 2 * acc_cols <= 256 ? 256 : 512;
  auto work = [&](int k) -> PairWork {
    if constexpr (DUAL) return pair_work(k, pair, pairs, tiles0, tiles1, second->extra);
    const int t = pair + k * pairs;
    return {0, t < tiles0 ? t : -1};
  };
  // parameters and tensor maps of the product that a piece of work belongs to
  auto params = [&](const PairWork& w) -> const GemmParams& {
    if constexpr (DUAL) return w.which ? second->p : p;
    else return p;
  };
  auto tensor_maps = [&](const PairWork& w) -> const PairMaps& {
    if constexpr (DUAL) return w.which ? second->m : maps;
    else return maps;
  };
  // the K steps of this CTA's part
  auto k_steps = [&](const GemmParams& q, int g, auto&& f) {
    if constexpr (SPLIT) {
      const int nkb = (q.K + BK - 1) / BK, hi = (int)((long long)nkb * (split + 1) / splits);
      for (int kb = (int)((long long)nkb * split / splits); kb < hi; ++kb)
        if (!f(kb * BK)) return;
    } else {
      for_each_k(q, g, f);
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      np::mbar_init(full_bar(s), 1);
      np::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      np::mbar_init(tfull_bar(a), 1);
      np::mbar_init(tempty_bar(a), 2 * EPI_WARPS);
    }
    for (int w = 0; w < EPI_WARPS; ++w) np::mbar_init(bar_base + 8u * (2 * STAGES + 4 + w), 1);
    *abort_flag = 0;
    np::mbar_fence_init();
  }
  if (threadIdx.x == 64) {   // while another warp sets up the barriers
    np::tma_prefetch_desc(&maps.A);
    np::tma_prefetch_desc(&maps.B);
    if (p.tma_c) np::tma_prefetch_desc(&maps.C);
    if (p.tma_c && p.C2) np::tma_prefetch_desc(&maps.C2);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     np::smem_u32((const void*)tmem_ptr_smem)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncwarp();
  np::tc_fence_before();
  cluster_sync();        // this CTA's and the peer's barriers and tensor memory are set up
  np::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  np::pdl_begin();
  auto epoch = [](const GemmParams& q) { return q.epoch + (q.epoch_base ? *q.epoch_base : 0); };

  // rows of the two 128-row blocks of an M block that carry data, as a mask (0: nothing to do, -1: gave up). Row-grouped
  // form: both blocks belong to the same group and arrive under the same flag (the caller's tables are made of pairs).
  auto tile_rows = [&](const GemmParams& q, const Tile& tl, int role) -> int {
    if (q.mode != 1) return 3;
    const int b0 = 2 * tl.m_blk;
    if (q.ready_flags) {
      const int fi = q.mblk_flag ? q.mblk_flag[b0] : 0;
      if (fi >= 0 && !np::wait_flag_ge(q.ready_flags + fi, epoch(q), q.flag_limit_ns, KID_GEMM, 120 + role)) {
        *abort_flag = 1;
        return -1;
      }
    }
    if (!q.mblk_rows) return 3;
    return (q.mblk_rows[b0] > 0 ? 1 : 0) | (b0 + 1 < (q.M + BM - 1) / BM && q.mblk_rows[b0 + 1] > 0 ? 2 : 0);
  };

  bool done = false;   // SPLIT: this epilogue warp's accumulator is complete
  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (one warp in each CTA, converged as above)
    int stage = 0;
    uint32_t phase = 0;
    bool live = true;
    for (int k = 0; live; ++k) {
      const PairWork wk = work(k);
      if (wk.t < 0) break;
      const GemmParams& q = params(wk);
      const PairMaps& tm = tensor_maps(wk);
      const uint32_t step_bytes = 2 * (A_BYTES + (q.b_mn ? (HN + 63) / 64 * 64 : HN) * BK * 2);   // of both CTAs
      const Tile tl = decode_tile<8>(wk.t, m_blocks(q), n_blocks(q));
      const int rows = __shfl_sync(0xffffffffu, lane == 0 ? tile_rows(q, tl, 0) : 0, 0);
      if (rows < 0) break;
      if (rows == 0) continue;
      const int m0 = tl.m_blk * TM + rank * BM;
      const int n0 = tl.n_blk * bn_out;
      long long goff = 0;
      if (q.mode == 1 && q.mblk_group) goff = (long long)q.mblk_group[2 * tl.m_blk] * q.group_stride_b;
      // SwiGLU: the leader's half of B is the gate tile, the peer's the up tile (another tensor, the same rows)
      const bool up = !DUAL && q.epilogue == 1 && rank;
      const CUtensorMap* bm = up ? &tm.B2 : &tm.B;
      const int nrow = n0 + (!DUAL && q.epilogue == 1 ? 0 : rank * HN);
      const int a_mn = q.a_mn, b_mn = q.b_mn, k_split = q.k_split;
      k_steps(q, tl.g, [&](int k0) -> bool {
        live = np::mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag, KID_GEMM, 11);
        if (!live) return false;
        if (np::elect_one()) {
          const uint32_t sA = smem_base + stage * STAGE_BYTES, sB = sA + A_BYTES;
          const uint32_t fb = peer_addr(full_bar(stage), lead);
          if (rank == 0) np::mbar_expect_tx(full_bar(stage), step_bytes);
          if (!a_mn) {
            tma_load_2d_pair(sA, &tm.A, fb, k0, m0);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c) tma_load_2d_pair(sA + c * (64 * BK * 2), &tm.A, fb, m0 + c * 64, k0);
          }
          if (!b_mn) {
            tma_load_2d_pair(sB, bm, fb, k0, (int)(nrow + goff));
          } else {
            const bool part2 = k_split && k0 >= k_split;
            const CUtensorMap* bk = part2 ? &tm.B2 : bm;
            const int kb = k0 + (int)goff - (part2 ? k_split : 0);
#pragma unroll
            for (int c = 0; c < (HN + 63) / 64; ++c) tma_load_2d_pair(sB + c * (64 * BK * 2), bk, fb, nrow + c * 64, kb);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        return true;
      });
    }
    // the leader's last commits have arrived here before this CTA may exit (a stage never used passes at once)
    for (int s = 0; s < STAGES; ++s) {
      if (!np::mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag, KID_GEMM, 15)) break;
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
    if (*abort_flag) __nanosleep(1000000);   // let copies already issued land before exit
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the leader's)
    if (rank == 0) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int k = 0;; ++k) {
        const PairWork wk = work(k);
        if (wk.t < 0) break;
        const GemmParams& q = params(wk);
        const uint32_t idesc = np::make_idesc(TM, BN, 1, 1, q.a_mn, q.b_mn);
        const uint64_t a_desc0 = operand_desc(smem_base, q.a_mn), b_desc0 = operand_desc(smem_base + A_BYTES, q.b_mn);
        const uint32_t a_step = k_step(q.a_mn), b_step = k_step(q.b_mn);
        const Tile tl = decode_tile<8>(wk.t, m_blocks(q), n_blocks(q));
        const int rows = __shfl_sync(0xffffffffu, lane == 0 ? tile_rows(q, tl, 1) : 0, 0);
        if (rows < 0) break;
        if (rows == 0) continue;
        if (count_k(q, tl.g) == 0) continue;
        if (!np::mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag, KID_GEMM, 12)) break;
        np::tc_fence_after();
        uint32_t tmem_d = tmem_base + (uint32_t)(acc * acc_cols);
        uint32_t accum = 0;
        const int parts = k_parts(q), nkb = parts > 1 ? count_k(q, tl.g) : 0;
        // 2 or 4 parts: the first K of the next one (a division per K step made the step half as long again)
        auto part_end = [&](int part) { return (int)((long long)nkb * (part + 1) >> (parts >> 1)) * BK; };
        int part = 0, next_k = parts > 1 ? part_end(0) : -1;
        k_steps(q, tl.g, [&](int k0) -> bool {
          if (PARTS && k0 == next_k) {   // the next part, in its own columns
            accum = 0;
            next_k = part_end(++part);
            tmem_d += BN;
            if (part == PER_BUFFER<BN>) {   // in the other buffer
              if (np::elect_one()) tc_commit_pair(tfull_bar(acc), lead);
              __syncwarp();
              if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
              if (!np::mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag, KID_GEMM, 17)) return false;
              np::tc_fence_after();
              tmem_d = tmem_base + (uint32_t)(acc * acc_cols);
            }
          }
          if (!np::mbar_wait_warp(full_bar(stage), phase, abort_flag, KID_GEMM, 13)) return false;
          np::tc_fence_after();
          if (np::elect_one()) {
            const uint64_t ad = a_desc0 + (uint32_t)(stage * (STAGE_BYTES >> 4)), bd = b_desc0 + (uint32_t)(stage * (STAGE_BYTES >> 4));
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              tc_mma_f16_pair(tmem_d, ad + kk * a_step, bd + kk * b_step, idesc, kk ? 1u : accum);
            tc_commit_pair(empty_bar(stage), lead);
          }
          __syncwarp();
          accum = 1;
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
          return true;
        });
        if (np::elect_one()) tc_commit_pair(tfull_bar(acc), lead);
        __syncwarp();
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
      if (*abort_flag) __nanosleep(1000000);
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    GluBar gb{bar_base + 8u * (2 * STAGES + 4 + warp - 2), 0u};
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int k = 0; !*abort_flag; ++k) {
      const PairWork wk = work(k);
      if (wk.t < 0) break;
      const GemmParams& q = params(wk);
      const PairMaps& tm = tensor_maps(wk);
      const Tile tl = decode_tile<8>(wk.t, m_blocks(q), n_blocks(q));
      const int rows = tile_rows(q, tl, 2);
      if (rows < 0) break;
      if (rows == 0) continue;
      const bool have_acc = count_k(q, tl.g) > 0;
      const bool mine = (rows >> rank) & 1;   // this CTA's 128-row block carries data
      const int parts = k_parts(q), buffers = parts > PER_BUFFER<BN> ? 2 : 1;
      if (have_acc) {
        if (!np::mbar_wait(tfull_bar(acc), acc_phase, abort_flag, KID_GEMM, 14)) break;
        if (buffers == 2 && !np::mbar_wait(tfull_bar(acc ^ 1), acc_phase ^ (uint32_t)acc, abort_flag, KID_GEMM, 18)) break;
        np::tc_fence_after();
      }
      if constexpr (SPLIT) { done = true; break; }   // one tile per cluster, finished below
      if (mine) {
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16), taddr = lanes + (uint32_t)(acc * acc_cols);
        const uint32_t stg = stg_base + (warp - 2) * STG_BYTES;
        const int row0 = tl.m_blk * TM + rank * BM + quarter * 32, n0 = tl.n_blk * bn_out;
        if (PARTS && parts > 1)
          add_parts<BN>(taddr, lanes + (uint32_t)((acc ^ 1) * acc_cols), parts, half, q.epilogue == 0 && q.tma_c && !q.out_f32);
        if (q.epilogue == 2) store_glu_bwd<BN>(q, &tm.C, &tm.C2, stg, gb, abort_flag, taddr, row0, lane, n0, half);
        else store_tile<BN>(q, &tm.C, &tm.C2, stg, taddr, tl.g, row0, lane, n0, half, have_acc);
      }
      if (have_acc) {
        np::tc_fence_before();
        __syncwarp();
        for (int b = 0; b < buffers; ++b) {
          if (lane == 0) arrive_cluster(peer_addr(tempty_bar(acc), lead));
          if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        }
      }
      if (q.done_counters && mine) {   // done_expected counts 128-row blocks
        const int fi = q.mblk_flag ? q.mblk_flag[2 * tl.m_blk] : 0;
        count_done(q, fi, EPI_WARPS * n_blocks(q) * q.done_expected[fi], epoch(q), lane);
      }
    }
    stage_drain(lane);
  }
  if constexpr (SPLIT) {
    __syncthreads();
    cluster_sync();      // every pair of the cluster has consumed its operand stages
    const int quarter = warp & 3, half = (warp - 2) >> 2, r = quarter * 32 + lane;
    const int W = BN / splits, per_half = W / 64;   // columns of a share; 32-column chunks of it per warp
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    auto slot = [&](int from, int c) {   // chunk c of the share sent by part `from`: [8 vectors][128 rows] of 16 bytes
      return smem_base + (uint32_t)(from * W * 512 + c * 8 * 2048 + r * 16);
    };
    if (done) {
      np::tc_fence_after();
      for (int d = 0; d < splits; ++d) {
        if (d == split) continue;
        for (int c = half * per_half; c < (half + 1) * per_half; ++c) {
          uint32_t v[32];
          np::tmem_ld32(taddr + d * W + c * 32, v);
          np::tmem_ld_wait();
          const uint32_t dst = peer_addr(slot(split, c), (uint32_t)(2 * d + rank));
#pragma unroll
          for (int i = 0; i < 8; ++i) st_cluster_v4(dst + i * 2048, v + 4 * i);
        }
      }
    }
    __syncwarp();
    cluster_sync();      // all shares have arrived
    if (done) {
      const Tile tl = decode_tile<8>(pair, m_blocks(p), n_blocks(p));
      const OutRow o = out_row(p, 0, tl.m_blk * TM + rank * BM + r);
      for (int c = half * per_half; c < (half + 1) * per_half; ++c) {
        uint32_t own[32];
        float sum[32];
        __syncwarp();
        np::tmem_ld32(taddr + split * W + c * 32, own);
        np::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[i] = 0.f;
        for (int d = 0; d < splits; ++d) {
          if (d == split) {
#pragma unroll
            for (int i = 0; i < 32; ++i) sum[i] += __uint_as_float(own[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float4 f;
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "r"(slot(d, c) + i * 2048) : "memory");
              sum[4 * i] += f.x; sum[4 * i + 1] += f.y; sum[4 * i + 2] += f.z; sum[4 * i + 3] += f.w;
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) own[i] = __float_as_uint(sum[i]);
        store_chunk(p, o, own, tl.n_blk * BN + split * W + c * 32);
      }
    }
    __syncwarp();
  }
  np::tc_fence_before();
  __syncthreads();
  cluster_sync();        // nothing of the peer reads or arrives here any more
  if (warp == 1) {
    np::tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

template <bool SPLIT, int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_pair_kernel(const __grid_constant__ PairMaps maps, const __grid_constant__ GemmParams p) {
  pair_body<SPLIT, BN, false>(maps, p, nullptr);
}
template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_pair2_kernel(const __grid_constant__ PairMaps maps, const __grid_constant__ GemmParams p,
                       const __grid_constant__ PairSecond second) {
  pair_body<false, BN, true>(maps, p, &second);
}

int g_num_sms = 0;

// Estimated time in us of a launch: a fixed part (setup, first loads, the drain of the last tile) and, per wave of tiles,
// the K steps one after the other plus what of the drain no MMA covers. Measured on B200 (launches of one kernel back to
// back in a graph): 256 x 256 output, K = 64 / 1024 / 4096: one-CTA 128 x 128 tiles 4.4 / 8.2 / 20.7, 128 x 256 tiles
// 5.2 / 9.4 / 22.8, pair with 256 columns 5.5 / 9.8 / 23.2, 192 columns 5.1 / 8.3 / 18.4, 128 columns 4.8 / 7.7 / 17.3, 256 with
// K in two parts 10.4 / 17.1 (K = 1024 / 4096), in four 10.6 / 14.0; with many SMs busy a K step is longer (2048 x 1024, K = 1024
// / 4096: 8.9 / 22.6, 10.1 / 27.8, 10.3 / 24.7, 9.4 / 21.4, 8.9 / 19.1).
struct TileCost { double fixed, step, drain; };
constexpr TileCost COST_128{4.3, 0.28, 0.4}, COST_256{5.0, 0.35, 0.3}, COST_PAIR{5.6, 0.30, 0.3}, COST_PAIR_192{5.3, 0.25, 0.3},
    COST_PAIR_128{5.2, 0.21, 0.3}, COST_SPLIT2{9.9, 0.30, 0.3}, COST_SPLIT4{11.7, 0.28, 0.3};
// Products of at most 64 rows. The few-row kernel: CTAs of 16 weight rows, each of which reads all of x again from the L2, so its
// time per CTA grows with the rows it is built for (8, 16, 32, 64) and, by the loads in flight, with K. The tile kernels pad to
// 128 rows but read x once per tile: with many columns they are bound by reading the weight. Fitted to 15 weights of 768 x 768 to
// 128256 x 2048 at 1 to 64 rows, DRAM-cold (us, few-row / best tile): 32000 x 2048: 8 rows 27.6 / 39.9, 16 39.9 / 39.9, 32 56 / 40,
// 64 92 / 40; 50264 x 768: 8 rows 27.6 / 29.7, 16 46 / 30; 6144 x 4096: 32 rows 27.7 / 32.9, 64 37.8 / 33.8; 4096 x 4096 and
// narrower outputs: few-row at every count (64 rows 27.6 / 31.8, 2048 x 5632 21.5 / 41.7).
inline double few_rows_cost(int M, int N, int K) {
  const double ctas = (N + 15) / 16;
  if (M <= 8) return 2.0 + ctas * (2.5e-3 + 4.0e-6 * K);
  if (M <= 16) return 2.0 + ctas * (8.0e-3 + 5.0e-6 * K);
  if (M <= 32) return 2.0 + ctas * (4.5e-3 + 10.5e-6 * K);
  return 2.0 + ctas * (9.0e-3 + 15.0e-6 * K);
}
inline double few_tiles_cost(double tiles, int N, int K) {   // tiles: estimate without the traffic; 5.0 TB/s of weight beside 5 us
  const double traffic = 5.0 + 2.0 * N * K / 5.0e6;
  return tiles > traffic ? tiles : traffic;
}
// Clusters of four and of eight CTAs that run at once (an SM pair per two CTAs, whole clusters within a GPC)
constexpr int CLUSTERS4 = 32, CLUSTERS8 = 14;
// Where the sum over K is cut (sum_rule): the estimates of the kernels that there were when the cuts were laid down
constexpr TileCost CUT_128{4.4, 0.37, 0.6}, CUT_256{5.3, 0.40, 0.3}, CUT_PAIR{6.0, 0.30, 0.3}, CUT_SPLIT2{9.3, 0.30, 0.3},
    CUT_SPLIT4{10.7, 0.30, 0.3};
// What the drain of a tile with K in parts takes beside that of a whole one: another read of the accumulator, and where the parts take
// both accumulator buffers, the part of the drain that otherwise runs under the next tile's products
inline double parts_drain(int parts, int bn) { return parts == 1 ? 0.0 : bn != 128 ? 1.5 : parts == 2 ? 0.2 : 0.8; }
}  // namespace

// ------------------------------------------------------------------ host side
static NpEncodeTiledFn g_encode = nullptr;
NpEncodeTiledFn np_get_encode_tiled() {
  if (g_encode) return g_encode;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  g_encode = (NpEncodeTiledFn)fn;
  return g_encode;
}

int np_make_tmap_2d(CUtensorMap* out, const void* base, int elt_bytes, uint64_t rows, uint64_t cols,
                    uint64_t ld, uint32_t box_cols, uint32_t box_rows) {
  NpEncodeTiledFn enc = np_get_encode_tiled();
  if (!enc) return -1;
  CUtensorMapDataType dt = elt_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                          : (elt_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32);
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * (uint64_t)elt_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

static int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return g_num_sms > 0 ? g_num_sms : 148;
}

// Output [planes][rows, cols] written in boxes of 32 rows x 128 bytes (128-byte swizzle)
static int make_tmap_out(CUtensorMap* out, const void* base, int f32, long long cols, long long rows, long long planes,
                         long long ld, long long plane_stride, int box_bytes = 128) {
  NpEncodeTiledFn enc = np_get_encode_tiled();
  if (!enc) return -1;
  const int es = f32 ? 4 : 2;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)planes};
  cuuint64_t strides[2] = {(cuuint64_t)(ld * es), (cuuint64_t)(plane_stride * es)};
  cuuint32_t box[3] = {(cuuint32_t)(box_bytes / es), 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base),
                   dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

// Tensor maps and kernel parameters of a launch with tiles of BN columns
template <int BN, bool PAIR>
static int prepare_gemm(const NpGemmArgs& a, int splits, int parts, PairMaps& m, CUtensorMap& tmAloc, CUtensorMap& tmBloc, GemmParams& p) {
  CUtensorMap &tmA = m.A, &tmB = m.B, &tmB2 = m.B2, &tmC = m.C, &tmC2 = m.C2;
  int rc;
  if (!a.a_mn) rc = np_make_tmap_2d(&tmA, a.A, 2, (uint64_t)a.a_rows, (uint64_t)a.K, (uint64_t)a.lda, BK, BM);
  else rc = np_make_tmap_2d(&tmA, a.A, 2, (uint64_t)a.a_rows, (uint64_t)a.M, (uint64_t)a.lda, 64, BK);
  if (rc) return 100 + rc;
  const uint32_t b_box_rows = (PAIR || a.epilogue == 1) ? BN / 2 : BN;
  if (!a.b_mn) rc = np_make_tmap_2d(&tmB, a.B, 2, (uint64_t)a.b_rows, (uint64_t)a.K, (uint64_t)a.ldb, BK, b_box_rows);
  else rc = np_make_tmap_2d(&tmB, a.B, 2, (uint64_t)a.b_rows, (uint64_t)a.N, (uint64_t)a.ldb, 64, BK);
  if (rc) return 200 + rc;
  tmB2 = tmB;
  if (a.epilogue == 1 || a.k_split > 0) {
    if (!a.b_mn) rc = np_make_tmap_2d(&tmB2, a.B2, 2, (uint64_t)a.b_rows, (uint64_t)a.K, (uint64_t)a.ldb, BK, b_box_rows);
    else rc = np_make_tmap_2d(&tmB2, a.B2, 2, (uint64_t)a.b_rows, (uint64_t)a.N, (uint64_t)a.ldb, 64, BK);
    if (rc) return 300 + rc;
  }
  if constexpr (!PAIR) {
    tmAloc = tmA;
    tmBloc = tmB;
  }
  p = GemmParams{};
  p.b_local_flag = a.b_local_flag - 1;
  // 32-byte stores need every (row, 32-column chunk) address 32-byte aligned; destinations behind peer_base are
  // allocations of the symmetric heap (256-byte aligned)
  static const bool st32_on = !(getenv("NPB200_ST32") != nullptr && getenv("NPB200_ST32")[0] == '0');
  const int per32 = a.out_f32 ? 8 : 16;   // elements of 32 bytes
  p.st32 = st32_on && (a.ldc % per32 == 0) && (a.group_stride_c % per32 == 0) &&
           (a.row_dst || (((uintptr_t)a.C) % 32 == 0 && (a.m_split == 0 || ((uintptr_t)a.C2) % 32 == 0)));
  p.st32_c2 = st32_on && a.ldc2 % 16 == 0 && a.N % 16 == 0 && ((uintptr_t)a.C2) % 32 == 0;
  if (a.push_src && a.push_n > 0) {
    if (a.push_n > 8 || (a.push_bytes & 15) || (((uintptr_t)a.push_src) & 15)) return 1;
    p.push_src = (const uint4*)a.push_src; p.push_vecs = a.push_bytes >> 4; p.push_n = a.push_n;
    p.push_ctr = a.push_ctr;
    for (int r = 0; r < a.push_n; ++r) { p.push_dst[r] = (uint4*)a.push_dst[r]; p.push_flag[r] = a.push_flag[r]; }
  }
  p.m_rot = a.m_rot; p.n_rot = a.n_rot; p.k_split = a.k_split; p.m_split = a.m_split;
  if (a.A_loc && !a.a_mn && a.a_loc_hi > a.a_loc_lo && a.a_loc_lo % BM == 0) {
    rc = np_make_tmap_2d(&tmAloc, a.A_loc, 2, (uint64_t)(a.a_loc_hi - a.a_loc_lo), (uint64_t)a.K, (uint64_t)a.lda_loc, BK, BM);
    if (rc) return 600 + rc;
    p.a_loc_lo = a.a_loc_lo; p.a_loc_hi = a.a_loc_hi;
  }
  if (a.B_loc && !a.b_mn && a.epilogue != 1 && a.b_loc_hi > a.b_loc_lo && a.b_loc_lo % b_box_rows == 0 &&
      (a.b_loc_hi - a.b_loc_lo) % b_box_rows == 0) {
    rc = np_make_tmap_2d(&tmBloc, a.B_loc, 2, (uint64_t)(a.b_loc_hi - a.b_loc_lo), (uint64_t)a.K, (uint64_t)a.ldb_loc, BK,
                         b_box_rows);
    if (rc) return 700 + rc;
    p.b_loc_lo = a.b_loc_lo; p.b_loc_hi = a.b_loc_hi;
  }
  p.C = a.C; p.C2 = a.C2; p.M = a.M; p.N = a.N; p.K = a.K; p.ldc = a.ldc; p.ldc2 = a.ldc2;
  p.bias = (a.epilogue == 0 && a.alpha != 0.f) ? a.bias : nullptr;
  p.a_mn = a.a_mn; p.b_mn = a.b_mn; p.out_f32 = a.out_f32; p.accumulate = a.accumulate;
  p.epilogue = a.epilogue; p.mode = a.mode; p.alpha = a.alpha;
  p.mblk_group = a.mblk_group; p.mblk_rows = a.mblk_rows; p.group_stride_b = a.group_stride_b;
  p.num_groups = a.num_groups; p.blocks_per_group = a.blocks_per_group; p.group_stride_c = a.group_stride_c;
  p.ready_flags = a.ready_flags; p.mblk_flag = a.mblk_flag; p.epoch = a.epoch;
  p.flag_limit_ns = a.flag_limit_ns ? a.flag_limit_ns : NP_WAIT_LIMIT_NS;
  p.row_dst = a.row_dst; p.peer_base = a.peer_base;
  p.done_counters = a.done_counters; p.done_expected = a.done_expected; p.done_flag_ptr = a.done_flag_ptr;
  p.local_push = a.local_push != 0;
  p.round_acc = a.round_acc != 0;
  p.Cin = a.Cin ? a.Cin : (a.accumulate ? a.C : nullptr);
  p.ldcin = a.Cin ? a.ldcin : a.ldc;
  p.epoch_base = a.epoch_base;
  p.b_ready_flags = a.b_ready_flags; p.b_rows_per_flag = a.b_rows_per_flag;

  // Rows that start on 16-byte boundaries are stored (and an accumulate source read) as whole vectors, other rows element by
  // element: an output of 1003 or 50257 columns has such rows. Destinations behind peer_base are symmetric-heap allocations.
  const int es = a.out_f32 ? 4 : 2;
  const long long groups = a.mode == 2 ? a.num_groups : 1;
  p.v16 = (a.ldc * es) % 16 == 0 && (groups <= 1 || (a.group_stride_c * es) % 16 == 0) &&
          (a.row_dst || ((uintptr_t)a.C & 15) == 0) && (a.m_split == 0 || ((uintptr_t)a.C2 & 15) == 0) &&
          (!p.Cin || (((uintptr_t)p.Cin & 15) == 0 && (p.ldcin * es) % 16 == 0));
  p.v16_c2 = a.C2 && ((uintptr_t)a.C2 & 15) == 0 && a.ldc2 % 8 == 0 && a.N % 8 == 0;   // the up half starts at column N
  // Plain outputs (dense rows, nothing added from memory, aligned) leave by TMA; peer-row tables, accumulation and other
  // alignments store from registers. The SwiGLU form needs both of its outputs aligned. So do rows whose length is no whole number
  // of 16 bytes: a tensor store rounds it up and fills with zeros, up to seven elements beside the output of a wider buffer.
  p.tma_c = p.v16 && (a.N * (long long)es) % 16 == 0 && !a.row_dst && !a.done_counters && !p.Cin && splits == 1 &&
            (a.epilogue != 1 || BN == 256) && a.ldc >= a.N && (a.epilogue != 1 || !a.C2 || p.v16_c2);
  tmC = tmA;
  tmC2 = tmA;
  if (a.epilogue == 2) {   // [d gate | d up] out, [gate | up] in: two planes of N columns each
    rc = make_tmap_out(&tmC, a.C, 0, a.N, a.M, 2, a.ldc, a.N, 64);
    if (!rc) rc = make_tmap_out(&tmC2, a.C2, 0, a.N, a.M, 2, a.ldc2, a.N, 64);
    if (rc) return 900 + rc;
  } else if (p.tma_c) {
    const long long gs = groups > 1 ? a.group_stride_c : a.ldc;
    rc = make_tmap_out(&tmC, a.C, a.out_f32, a.N, a.m_split > 0 ? a.m_split : a.M, groups, a.ldc, gs);
    if (!rc && a.m_split > 0) rc = make_tmap_out(&tmC2, a.C2, a.out_f32, a.N, a.M - a.m_split, groups, a.ldc, gs);
    if (!rc && a.epilogue == 1 && a.C2) rc = make_tmap_out(&tmC2, a.C2, 0, a.N, a.M, 2, a.ldc2, a.N);
    if (rc) return 800 + rc;
  }
  p.splits = splits;
  p.parts = parts;
  return 0;
}

template <int BN, bool PAIR>
constexpr int gemm_smem() {
  constexpr int STAGES = PAIR ? pair_stages<BN>() : BN == 256 ? 4 : 6;
  return STAGES * (PAIR ? pair_stage_bytes<BN>() : BM * BK * 2 + BN * BK * 2) + EPI_WARPS * STG_BYTES + 1024 + 256;
}

template <int BN, bool PAIR>
static int launch_gemm(const NpGemmArgs& a, cudaStream_t stream, int splits = 1, int parts = 1) {
  PairMaps m;
  CUtensorMap tmAloc, tmBloc;
  GemmParams p;
  const int rc = prepare_gemm<BN, PAIR>(a, splits, parts, m, tmAloc, tmBloc, p);
  if (rc) return rc;
  constexpr int SMEM = gemm_smem<BN, PAIR>(), STAGES = BN == 256 ? 4 : 6;
  static_assert(SMEM <= 227 * 1024, "shared memory budget");
  static NpPerDeviceOnce attr_once;
  bool& attr_set = *attr_once.slot();
  if (!attr_set) {
    cudaError_t e;
    if constexpr (PAIR) {
      e = cudaFuncSetAttribute(gemm_bf16_pair_kernel<false, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
      if constexpr (BN == 256)
        if (e == cudaSuccess)
          e = cudaFuncSetAttribute(gemm_bf16_pair_kernel<true, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    } else e = cudaFuncSetAttribute(gemm_bf16_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return 400 + (int)e;
    attr_set = true;
  }
  const int cap = a.max_ctas > 0 ? a.max_ctas : num_sms();
  const int bn_out = a.epilogue == 1 ? BN / 2 : BN, tm = PAIR ? 2 * BM : BM;
  const long long tiles = (long long)((a.M + tm - 1) / tm) * ((a.N + bn_out - 1) / bn_out) * (a.mode == 2 ? a.num_groups : 1);
  if (tiles <= 0) return 0;   // K-grouped form without groups
  const bool busy = 2.0 * a.M * a.N * a.K > 2e10;   // 15 us and more
  if constexpr (PAIR) {
    const long long pairs = tiles < cap / 2 ? tiles : cap / 2;
    if (pairs <= 0) return 1;   // the dispatch gives launches of one CTA to the other kernel
    const dim3 grid((unsigned)(splits > 1 ? tiles * 2 * splits : 2 * pairs));
    auto kern = gemm_bf16_pair_kernel<false, BN>;
    if constexpr (BN == 256)
      if (splits > 1) kern = gemm_bf16_pair_kernel<true, BN>;
    const cudaError_t e =
        np_launch_if(busy, kern, grid, GEMM_THREADS, SMEM, stream, 2 * splits, m, p);
    if (e != cudaSuccess) return 500 + (int)e;
  } else {
    const int grid = (int)(tiles < cap ? tiles : cap);
    np_launch_if(busy, gemm_bf16_kernel<BN, STAGES>, grid, GEMM_THREADS, SMEM, stream, 1, m.A, m.B, m.B2, tmAloc, tmBloc, m.C, m.C2, p);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

int np_skinny_linear(const void* x, long long ldx, const void* w, long long ldw, int M, int N, int K, void* out, long long ldo,
                     int out_f32, float alpha, const float* bias, const void* cin, long long ldcin, cudaStream_t stream);

// The tensor-map encode is a driver call: make sure this host thread (e.g. an autograd worker that has not touched the runtime
// yet) has the device's primary context bound.
static bool bind_context() {
  static thread_local bool bound = false;
  if (!bound) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess || cudaFree(nullptr) != cudaSuccess) return false;
    bound = true;
  }
  return true;
}
static int check_gemm(const NpGemmArgs& a) {
  if (a.k_split < 0 || a.m_split < 0 || (a.k_split > 0 && (!a.b_mn || a.mode == 2 || a.epilogue != 0 || a.k_split % BK)) ||
      (a.m_split > 0 && (a.row_dst || a.epilogue != 0 || a.m_split % 256 || a.m_split >= a.M || (a.Cin && a.Cin != a.C))))
    return 1;
  if (a.epilogue == 2 && (a.mode == 2 || a.out_f32 || a.accumulate || a.Cin || a.row_dst || a.done_counters || !a.C2 || a.N % 8 ||
                          a.ldc % 8 || a.ldc2 % 8 || (((uintptr_t)a.C | (uintptr_t)a.C2) & 15)))
    return 1;
  if ((a.lda % 8) || (a.ldb % 8) || (((uintptr_t)a.A) & 15) || (((uintptr_t)a.B) & 15)) return 1;
  if (a.pair_bn != 0 && a.pair_bn != 128 && a.pair_bn != 192 && a.pair_bn != 256) return 1;
  return 0;
}

// Which kernel a product runs on: the few-row kernel, one CTA per tile of `bn` columns, or pairs with tiles of `bn` columns. K in
// `splits` parts over a cluster, or in `parts` that one pair sums in turn: the same sums, added in the same order.
struct GemmChoice {
  bool few, pair;
  int bn, splits, parts;
  double cost;   // estimate in us
};
// Tiles of tm x tn and K steps of a tile. Grouped forms by the room of their regions, as which rows arrive is not known here; an estimate
// from the mean rows per expert chose worse (the six GEMMs of an expert layer 525 -> 609 us at 4096 tokens, 174 -> 208 at 512).
static long long tiles_of(const NpGemmArgs& a, int tm, int tn) {
  return (long long)((a.M + tm - 1) / tm) * ((a.N + tn - 1) / tn) * (a.mode == 2 ? a.num_groups : 1);
}
static double tile_steps(const NpGemmArgs& a) { return a.mode == 2 ? 2.0 * a.blocks_per_group : (a.K + BK - 1) / BK; }
static double operations(const NpGemmArgs& a) { return tiles_of(a, BM, BM) * 2.0 * BM * BM * BK * tile_steps(a); }

// What a launch allows: forms for the pair kernel, and K in parts (dense plain outputs). The pair kernel takes the forms without
// peer-arrival flags on B, pushes or split operands; row-grouped launches only when their tables come in pairs of 128-row blocks
// (`paired`).
struct GemmForms {
  bool plain, pair, split;
  int sms;
};
static GemmForms forms_of(const NpGemmArgs& a) {
  GemmForms f;
  f.sms = a.max_ctas > 0 ? a.max_ctas : num_sms();
  f.plain = !a.b_ready_flags && !a.push_src && !a.A_loc && !a.B_loc && a.m_rot == 0 && a.n_rot == 0 &&
            (a.mode == 1 ? a.paired != 0 : !a.row_dst && !a.ready_flags && !a.done_counters);
  f.pair = f.plain && f.sms >= 2;   // a pair needs two CTAs
  // a SwiGLU gradient of a rounded dh: the sum that dh as a product of its own has
  f.split = f.plain && a.k_split == 0 && a.m_split == 0 && a.mode == 0 && (a.epilogue == 0 || (a.epilogue == 2 && a.round_acc)) &&
            (a.K + BK - 1) / BK >= 8 && a.max_ctas == 0 && a.M > 128;
  return f;
}
static double launch_cost(const NpGemmArgs& a, const TileCost& t, int tm, int tn, int units, int splits) {
  const long long n = tiles_of(a, tm, tn);
  const double waves = (double)((n + units - 1) / units), steps = tile_steps(a);
  // tiles of a persistent CTA follow one another; a cluster that splits K starts anew for every tile
  return splits == 1 ? t.fixed + waves * (steps * t.step + t.drain) : waves * (t.fixed + steps / splits * t.step + t.drain);
}

// How a product's sum over K is formed where the caller asks for no tile: by the few-row kernel, whole, or in 2 or 4 parts that are
// added in order. A rule of the product's own sizes, apart from the choice of the kernel that runs it: a product has the same bits on
// every tile, alone or beside another one in a launch. Other cuts round differently, and after a layer or two of bf16 results that
// is more than the last bits: a training step whose gradients were summed whole instead of in parts moved its loss by 2e-3.
struct SumRule {
  bool few;
  int parts;
};
static SumRule sum_rule(const NpGemmArgs& a, const GemmForms& f) {
  double best = 1e30;
  int parts = 1;
  auto take = [&](const TileCost& t, int tm, int tn, int units, int n) {
    const double cost = launch_cost(a, t, tm, tn, units, n);
    if (cost < best) { best = cost; parts = n; }
  };
  const int n256 = a.epilogue == 1 ? 128 : 256;
  if (a.epilogue != 1 && a.bn != 256) take(CUT_128, 128, 128, f.sms, 1);
  take(CUT_256, 128, n256, f.sms, 1);
  if (f.pair && a.M > 128) take(CUT_PAIR, 256, n256, f.sms / 2, 1);
  if (f.split && a.split == 0 && f.sms >= 128) {
    take(CUT_SPLIT2, 256, 256, CLUSTERS4, 2);
    take(CUT_SPLIT4, 256, 256, CLUSTERS8, 4);
  }
  // A few rows of a K-major product: the kernel that streams the weight once through all SMs (skinny.cu), unless a tile kernel
  // is expected to be faster. `mt`, `bn`, `split` and `pair_bn` ask for a tile kernel.
  const bool few = a.M <= 64 && a.mode == 0 && a.epilogue == 0 && !a.a_mn && !a.b_mn && f.plain && a.K > 0 && a.K % 8 == 0 &&
                   a.bn == 0 && a.mt == 0 && a.split == 0 && a.pair_bn == 0 && a.max_ctas == 0 && a.alpha != 0.f &&
                   few_rows_cost(a.M, a.N, a.K) <= few_tiles_cost(best, a.N, a.K);
  return {few, parts};
}

// The kernel with the lowest estimate (TileCost) among those that form the sum as the rule says
static GemmChoice choose_gemm(const NpGemmArgs& a) {
  const GemmForms f = forms_of(a);
  const int bn_asked = a.epilogue == 1 ? 256 : a.bn, pbn_asked = a.epilogue == 1 ? 0 : a.pair_bn;
  const bool split_asked = f.split && a.epilogue == 0 && (a.split == 2 || a.split == 4);
  GemmChoice c{false, false, bn_asked == 256 ? 256 : 128, 1, 1, 1e30};
  if (f.pair && bn_asked != 128 && (a.mt == 2 || pbn_asked != 0 || (a.mt == 0 && split_asked))) {
    c.pair = true;   // asked for
    c.bn = pbn_asked == 0 || (split_asked && pbn_asked != 128) ? 256 : pbn_asked;
    if (split_asked) (c.bn == 128 ? c.parts : c.splits) = a.split;
  } else if (bn_asked == 0 || (bn_asked == 256 && a.mt == 0)) {
    const SumRule rule = a.mt == 0 ? sum_rule(a, f) : SumRule{false, 1};
    auto take = [&](TileCost t, int tm, int tn, int units, bool pair, int bn, int splits, int parts) {
      t.drain += parts_drain(parts, bn);
      const double cost = launch_cost(a, t, tm, tn, units, splits);
      if (cost < c.cost) c = GemmChoice{false, pair, bn, splits, parts, cost};
    };
    const int n256 = a.epilogue == 1 ? 128 : 256;
    if (rule.parts == 1) {
      if (bn_asked == 0) take(COST_128, 128, 128, f.sms, false, 128, 1, 1);
      take(COST_256, 128, n256, f.sms, false, 256, 1, 1);
      if (f.pair && a.M > 128 && a.mt == 0) {
        take(COST_PAIR, 256, n256, f.sms / 2, true, 256, 1, 1);
        if (bn_asked == 0) {
          take(COST_PAIR_192, 256, 192, f.sms / 2, true, 192, 1, 1);
          take(COST_PAIR_128, 256, 128, f.sms / 2, true, 128, 1, 1);
        }
      }
    } else {
      if (bn_asked == 0) take(COST_PAIR_128, 256, 128, f.sms / 2, true, 128, 1, rule.parts);
      if (a.epilogue == 0) {
        if (rule.parts == 2) take(COST_SPLIT2, 256, 256, CLUSTERS4, true, 256, 2, 1);
        else take(COST_SPLIT4, 256, 256, CLUSTERS8, true, 256, 4, 1);
      }
    }
    c.few = rule.few;
  }
  return c;
}

// C[M,N] (+)= alpha * A * B^T with the operand layouts described in NpGemmArgs.
// Returns 0 or a launch/setup error; device-side problems are reported via np_status_read.
NP_API int np_gemm_bf16(const NpGemmArgs* args, void* stream) {
  const NpGemmArgs& a = *args;
  if (a.M <= 0 || a.N <= 0) return 0;
  if (!bind_context()) return 2;
  if (check_gemm(a)) return 1;
  const GemmChoice c = choose_gemm(a);
  if (c.few)
    return np_skinny_linear(a.A, a.lda, a.B, a.ldb, a.M, a.N, a.K, a.C, a.ldc, a.out_f32, a.alpha, a.bias,
                            a.Cin ? a.Cin : (a.accumulate ? a.C : nullptr), a.Cin ? a.ldcin : a.ldc, (cudaStream_t)stream);
  if (c.pair)
    return c.bn == 128   ? launch_gemm<128, true>(a, (cudaStream_t)stream, 1, c.parts)
           : c.bn == 192 ? launch_gemm<192, true>(a, (cudaStream_t)stream)
                         : launch_gemm<256, true>(a, (cudaStream_t)stream, c.splits);
  if (c.bn == 256) return launch_gemm<256, false>(a, (cudaStream_t)stream);
  return launch_gemm<128, false>(a, (cudaStream_t)stream);
}

template <int BN>
static int launch_gemm2(const NpGemmArgs& a, int parts_a, const NpGemmArgs& b, int parts_b, int extra, cudaStream_t stream) {
  PairMaps m;
  GemmParams p;
  PairSecond second;
  CUtensorMap unused;
  int rc = prepare_gemm<BN, true>(a, 1, parts_a, m, unused, unused, p);
  if (!rc) rc = prepare_gemm<BN, true>(b, 1, parts_b, second.m, unused, unused, second.p);
  if (rc) return rc;
  second.extra = extra;
  constexpr int SMEM = gemm_smem<BN, true>();
  static NpPerDeviceOnce attr_once;
  bool& attr_set = *attr_once.slot();
  if (!attr_set) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_bf16_pair2_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return 400 + (int)e;
    attr_set = true;
  }
  const long long n = tiles_of(a, 256, BN) + tiles_of(b, 256, BN), pairs = n < num_sms() / 2 ? n : num_sms() / 2;
  const bool busy = operations(a) + operations(b) > 2e10;   // 15 us and more
  cudaError_t e = np_launch_if(busy, gemm_bf16_pair2_kernel<BN>, dim3((unsigned)(2 * pairs)), GEMM_THREADS, SMEM, stream, 2, m, p, second);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

// Two independent products: in one launch where both run on pairs of CTAs and are expected to take less time that way, else one after
// the other, with the same bits. A product grouped by rows may wait for arrivals and push; what the other one reads has to be there at
// launch. `pair_bn` of the first asks for one launch with tiles of that many columns (128 where a sum has four parts), `split` 1 or
// `mt` 2 of the first for two launches.
NP_API int np_gemm_bf16_two(const NpGemmArgs* first, const NpGemmArgs* second, void* stream) {
  const NpGemmArgs &a = *first, &b = *second;
  auto separate = [&] {
    const int rc = np_gemm_bf16(first, stream);
    return rc ? rc : np_gemm_bf16(second, stream);
  };
  auto pairable = [](const NpGemmArgs& g) {
    return g.M > 128 && g.N > 0 && g.K > 0 && g.epilogue != 1 && !g.b_ready_flags && !g.push_src && !g.A_loc && !g.B_loc &&
           g.m_rot == 0 && g.n_rot == 0 && g.bn == 0 && g.mt == 0 && g.split == 0 && g.max_ctas == 0 &&
           (g.mode == 1 ? g.paired != 0 : !g.row_dst && !g.ready_flags && !g.done_counters) && (g.mode != 2 || g.num_groups > 0);
  };
  const int units = num_sms() / 2;
  // Long products run at the power limit: SMs that idle let the others run faster, so there is nothing to fill (us, two launches /
  // one: 4096 tokens, 2048 x 11264, 3.8e11 operations 261 / 256; 2048 x 32000, 1.1e12 799 / 846).
  const bool long_run = operations(a) + operations(b) > 6e11 && a.pair_bn == 0;
  if (!pairable(a) || !pairable(b) || b.pair_bn != 0 || units < 1 || long_run) return separate();
  if (!bind_context()) return 2;
  if (check_gemm(a) || check_gemm(b)) return 1;
  // the longer contraction first
  const bool swap = tile_steps(b) > tile_steps(a);
  const NpGemmArgs &x = swap ? b : a, &y = swap ? a : b;
  const double sx = tile_steps(x), sy = tile_steps(y);
  const int px = sum_rule(x, forms_of(x)).parts, py = sum_rule(y, forms_of(y)).parts;
  const bool wide = px <= 2 && py <= 2;   // four parts: two accumulators a buffer
  const int asked = a.pair_bn != 0 && !wide ? 128 : a.pair_bn;
  double best = a.pair_bn != 0 ? 1e30 : choose_gemm(a).cost + choose_gemm(b).cost;
  int bn = 0, extra = 0;
  auto take = [&](const TileCost& t, int cols) {   // the pair with the most to do
    if (asked != 0 && asked != cols) return;
    const int nx = (int)tiles_of(x, 256, cols), ny = (int)tiles_of(y, 256, cols);
    const int pairs = nx + ny < units ? nx + ny : units;
    const double cx = sx * t.step + t.drain + parts_drain(px, cols), cy = sy * t.step + t.drain + parts_drain(py, cols);
    const int ex = (int)(cx / cy);
    // pair 0 has one of the first product's tiles more than pair r; behind each, the others have as much or less
    const int r = nx % pairs, slack = pairs - r, rest = ny - (r == 0 ? 0 : ex < (ny + slack - 1) / slack ? ex * slack : ny);
    auto dealt = [&](int at) { return rest > at ? (rest - at - 1) / pairs + 1 : 0; };
    const double at_0 = ((nx + pairs - 1) / pairs) * cx + dealt(r == 0 ? 0 : slack) * cy;
    const int before = ex < (ny + slack - 1) / slack ? ex : (ny + slack - 1) / slack;
    const double at_r = r == 0 ? 0 : (nx / pairs) * cx + (before + dealt(0)) * cy;
    const double most = at_0 > at_r ? at_0 : at_r;
    if (t.fixed + most < best) { best = t.fixed + most; bn = cols; extra = ex; }
  };
  if (wide) {
    take(COST_PAIR, 256);
    take(COST_PAIR_192, 192);
  }
  take(COST_PAIR_128, 128);
  cudaStream_t st = (cudaStream_t)stream;
  return bn == 256   ? launch_gemm2<256>(x, px, y, py, extra, st)
         : bn == 192 ? launch_gemm2<192>(x, px, y, py, extra, st)
         : bn == 128 ? launch_gemm2<128>(x, px, y, py, extra, st)
                     : separate();
}

NP_API int np_status_read(int* out8) {
  return (int)cudaMemcpyFromSymbol(out8, g_np_status, sizeof(int) * 8);
}
// Per-SM communication time in ns accumulated since the last reset (see account_interval): copies NP_MAX_SMS
// values into `out_ns` and, when `reset` is set, zeroes the counters. Synchronises the device.
NP_API int np_wait_stats_read(unsigned long long* out_ns, int reset) {
  cudaError_t e = cudaMemcpyFromSymbol(out_ns, g_np_wait_ns, sizeof(unsigned long long) * NP_MAX_SMS);
  if (e != cudaSuccess) return (int)e;
  if (reset) {
    static const unsigned long long z[NP_MAX_SMS] = {0};
    e = cudaMemcpyToSymbol(g_np_wait_ns, z, sizeof(z));
  }
  return (int)e;
}
NP_API int np_wait_stats_slots() { return NP_MAX_SMS; }
NP_API int np_status_clear() {
  int z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  return (int)cudaMemcpyToSymbol(g_np_status, z, sizeof(z));
}
NP_API int np_num_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}
