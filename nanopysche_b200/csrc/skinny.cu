// Kernels for a few rows at a time (token generation): a linear layer of up to 64 rows, and attention of a few query rows
// against a KV cache with the new keys and values appended in the same pass. Both stream one large operand (the weight,
// the cache) through the chip once and are bound by that traffic and by launch latency; tensor-memory tiles of 128 rows
// would leave most of the chip idle (a 2048 x 2048 weight is 16 tiles).
#include "common.cuh"
#include "args.h"

namespace {

// ------------------------------------------------------------------------------------------------------- linear layer
// y[M, N] = alpha * x[M, K] w[N, K]^T (+ bias) (+ cin). A CTA owns 16 weight rows, its eight warps share K in units of 64:
// every lane reads 32 contiguous bytes of a weight row per unit, four lanes a whole 128-byte line. mma.sync m16n8k16 with
// the weight rows as the M side; which 16 of the 64 elements form one k step is free as long as both operands agree, so a
// lane's 16 elements feed four MMAs without any shuffle. The warps' partial sums meet in shared memory in warp order
// (deterministic).
struct SkinnyParams {
  const __nv_bfloat16* x; const __nv_bfloat16* w;
  long long ldx, ldw;
  int M, N, K;
  void* out; long long ldo; int out_f32;
  float alpha;
  const float* bias;
  const void* cin; long long ldcin;
};

__device__ __forceinline__ void mma16816(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 bytes of a row, or zeros past the end of K (K is a multiple of 8)
__device__ __forceinline__ uint4 ld16(const __nv_bfloat16* row, int k, int K) {
  return k < K ? *reinterpret_cast<const uint4*>(row + k) : make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ uint4 ld16_stream(const __nv_bfloat16* row, int k, int K) {   // read once: do not keep in L1
  uint4 v = make_uint4(0, 0, 0, 0);
  if (k < K)
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(row + k));
  return v;
}

constexpr int SK_WARPS = 8;

// MT: tiles of 8 rows of x (M <= 8 MT); U: units of 64 in flight per warp
template <int MT, int U>
__global__ void __launch_bounds__(SK_WARPS * 32)
skinny_linear_kernel(const SkinnyParams p) {
  __shared__ float red[SK_WARPS][MT][16][8];
  np::pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16;
  const int r0 = n0 + g < p.N ? n0 + g : p.N - 1, r1 = n0 + 8 + g < p.N ? n0 + 8 + g : p.N - 1;
  const __nv_bfloat16* w0 = p.w + (long long)r0 * p.ldw;
  const __nv_bfloat16* w1 = p.w + (long long)r1 * p.ldw;
  const __nv_bfloat16* xr[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const int row = m * 8 + g;
    xr[m] = p.x + (long long)(row < p.M ? row : p.M - 1) * p.ldx;   // rows past the end are computed and not stored
  }
  float acc[MT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
  const int units = (p.K + 63) / 64;
  for (int u0 = warp; u0 < units; u0 += SK_WARPS * U) {
    uint4 a[U][4];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = (u0 + i * SK_WARPS) * 64 + t * 16;   // units past the end read as zeros
      a[i][0] = ld16_stream(w0, k, p.K); a[i][1] = ld16_stream(w0, k + 8, p.K);
      a[i][2] = ld16_stream(w1, k, p.K); a[i][3] = ld16_stream(w1, k + 8, p.K);
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int k = (u0 + i * SK_WARPS) * 64 + t * 16;
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const uint4 b0 = ld16(xr[m], k, p.K), b1 = ld16(xr[m], k + 8, p.K);
        mma16816(acc[m], a[i][0].x, a[i][2].x, a[i][0].y, a[i][2].y, b0.x, b0.y);
        mma16816(acc[m], a[i][0].z, a[i][2].z, a[i][0].w, a[i][2].w, b0.z, b0.w);
        mma16816(acc[m], a[i][1].x, a[i][3].x, a[i][1].y, a[i][3].y, b1.x, b1.y);
        mma16816(acc[m], a[i][1].z, a[i][3].z, a[i][1].w, a[i][3].w, b1.z, b1.w);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    red[warp][m][g][2 * t] = acc[m][0]; red[warp][m][g][2 * t + 1] = acc[m][1];
    red[warp][m][g + 8][2 * t] = acc[m][2]; red[warp][m][g + 8][2 * t + 1] = acc[m][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < MT * 128; i += SK_WARPS * 32) {
    const int n = i & 15, m = i >> 4;                    // 16 neighbouring threads store 16 neighbouring columns
    const int col = n0 + n;
    if (m >= p.M || col >= p.N) continue;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < SK_WARPS; ++q) v += red[q][m >> 3][n][m & 7];
    v *= p.alpha;
    if (p.bias) v += p.bias[col];
    if (p.out_f32) {
      if (p.cin) v += ((const float*)p.cin)[(long long)m * p.ldcin + col];
      ((float*)p.out)[(long long)m * p.ldo + col] = v;
    } else {
      if (p.cin) v += __bfloat162float(((const __nv_bfloat16*)p.cin)[(long long)m * p.ldcin + col]);
      ((__nv_bfloat16*)p.out)[(long long)m * p.ldo + col] = __float2bfloat16(v);
    }
  }
}

// ---------------------------------------------------------------------------------------------- attention with a KV cache
// o = softmax(q [k_cache | k_new]^T) [v_cache | v_new] for a few query rows, and - when asked for - the concatenated cache
// itself, written from the very registers that the products read: a key or value crosses the chip once, where a separate
// concatenation reads and writes the whole cache first. One cluster of CTAs per (batch, KV head) shares the keys; a warp
// takes 32 / (HD / 8) keys per load (16 bytes a lane), every group of HD / 8 lanes keeps its own running maximum, sum and
// output for the R = n_rep * Sq query rows, and these meet in a fixed order: lanes, warps, then the CTAs of the cluster
// through distributed shared memory.
struct DecodeParams {
  const __nv_bfloat16* q; long long q_sb, q_ss, q_sh;
  const __nv_bfloat16* kc; const __nv_bfloat16* vc; long long kc_sb, kc_ss, kc_sh, vc_sb, vc_ss, vc_sh;   // cache
  const __nv_bfloat16* kn; const __nv_bfloat16* vn; long long kn_sb, kn_ss, kn_sh, vn_sb, vn_ss, vn_sh;   // new rows
  __nv_bfloat16* ko; __nv_bfloat16* vo;     // concatenated [B, past + fresh, Hkv, HD], or nullptr
  __nv_bfloat16* o;                         // [B, Sq, Hq, HD]
  int B, Sq, Hq, Hkv, past, fresh, causal;
  float scale_log2;
};

__device__ __forceinline__ float ex2a(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  const float2 a = np::unpack_bf16(v.x), b = np::unpack_bf16(v.y), c = np::unpack_bf16(v.z), d = np::unpack_bf16(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t cta) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(np::smem_u32(p)), "r"(cta));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

constexpr int DC_WARPS = 8;

template <int HD, int R>
__global__ void __launch_bounds__(DC_WARPS * 32, R <= 2 ? 2 : 1)
decode_attn_kernel(const DecodeParams p) {
  constexpr int L = HD / 8, KPW = 32 / L, U = 2, STEP = DC_WARPS * KPW * U;
  __shared__ float s_m[DC_WARPS][R], s_l[DC_WARPS][R], s_acc[DC_WARPS][R][HD];
  __shared__ float c_m[R], c_l[R], c_acc[R][HD];
  np::pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / L, d0 = (lane % L) * 8;
  const int part = blockIdx.x, parts = gridDim.x, h = blockIdx.y, b = blockIdx.z;   // a cluster spans grid.x
  const int n_rep = p.Hq / p.Hkv, rows = n_rep * p.Sq, total = p.past + p.fresh;
  const int lo = (int)((long long)total * part / parts), hi = (int)((long long)total * (part + 1) / parts);
  float q[R][8], acc[R][8], m[R], l[R];
  int last[R];                                             // last visible key of a row
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int rr = r < rows ? r : rows - 1, rep = rr / p.Sq, i = rr % p.Sq;
    unpack8(*reinterpret_cast<const uint4*>(p.q + b * p.q_sb + i * p.q_ss + (long long)(h * n_rep + rep) * p.q_sh + d0), q[r]);
#pragma unroll
    for (int e = 0; e < 8; ++e) { q[r][e] *= p.scale_log2; acc[r][e] = 0.f; }
    m[r] = -INFINITY; l[r] = 0.f;
    last[r] = p.causal ? total - p.Sq + i : total - 1;
  }
  // Keys [k0, k1) of one source (row k0 at kp / vp), the first of them being key `key0` of the sequence. Two keys per lane
  // group at a time, the next two already on their way.
  auto attend = [&](const __nv_bfloat16* kp, const __nv_bfloat16* vp, long long kss, long long vss, int n, int key0) {
    int at = warp * (KPW * U) + sub;                       // this lane group's first key
    kp += at * kss + d0;
    vp += at * vss + d0;
    const long long kstep = STEP * kss, vstep = STEP * vss, ku = KPW * kss, vu = KPW * vss;
    __nv_bfloat16* ko = p.ko ? p.ko + (((long long)b * total + key0 + at) * p.Hkv + h) * HD + d0 : nullptr;
    __nv_bfloat16* vo = p.ko ? p.vo + (((long long)b * total + key0 + at) * p.Hkv + h) * HD + d0 : nullptr;
    const long long ou = (long long)KPW * p.Hkv * HD, ostep = (long long)STEP * p.Hkv * HD;
    uint4 kn[U], vn[U];
    auto fetch = [&]() {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        kn[u] = vn[u] = make_uint4(0, 0, 0, 0);
        if (at + u * KPW < n) {
          kn[u] = *reinterpret_cast<const uint4*>(kp + u * ku);
          vn[u] = *reinterpret_cast<const uint4*>(vp + u * vu);
        }
      }
    };
    fetch();
    for (int base = warp * (KPW * U); base < n; base += STEP) {   // the same trip count for the warp
      uint4 kv[U], vv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) { kv[u] = kn[u]; vv[u] = vn[u]; }
      const int cur = at;
      at += STEP;
      kp += kstep;
      vp += vstep;
      fetch();
      float s[U][R];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = cur + u * KPW < n;
        if (ko && in) {
          *reinterpret_cast<uint4*>(ko + u * ou) = kv[u];
          *reinterpret_cast<uint4*>(vo + u * ou) = vv[u];
        }
        float f[8];
        unpack8(kv[u], f);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float v = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) v = fmaf(q[r][e], f[e], v);
#pragma unroll
          for (int x = L / 2; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
          s[u][r] = (in && key0 + cur + u * KPW <= last[r]) ? v : -INFINITY;
        }
      }
      if (ko) { ko += ostep; vo += ostep; }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float mx = m[r];
#pragma unroll
        for (int u = 0; u < U; ++u) mx = fmaxf(mx, s[u][r]);
        const float mu = mx == -INFINITY ? 0.f : mx;
        const float c = ex2a(m[r] - mu);
        m[r] = mx;
        l[r] *= c;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[r][e] *= c;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          s[u][r] = ex2a(s[u][r] - mu);
          l[r] += s[u][r];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float f[8];
        unpack8(vv[u], f);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[r][e] = fmaf(s[u][r], f[e], acc[r][e]);
      }
    }
  };
  const int c_hi = hi < p.past ? hi : p.past, f_lo = lo > p.past ? lo : p.past;
  if (lo < c_hi)
    attend(p.kc + b * p.kc_sb + lo * p.kc_ss + h * p.kc_sh, p.vc + b * p.vc_sb + lo * p.vc_ss + h * p.vc_sh, p.kc_ss, p.vc_ss,
           c_hi - lo, lo);
  if (f_lo < hi)
    attend(p.kn + b * p.kn_sb + (f_lo - p.past) * p.kn_ss + h * p.kn_sh, p.vn + b * p.vn_sb + (f_lo - p.past) * p.vn_ss + h * p.vn_sh,
           p.kn_ss, p.vn_ss, hi - f_lo, f_lo);
  // the groups of lanes, then the warps, then the CTAs of the cluster
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int x = L; x < 32; x <<= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[r], x), lo2 = __shfl_xor_sync(0xffffffffu, l[r], x);
      const float mx = fmaxf(m[r], mo), mu = mx == -INFINITY ? 0.f : mx;
      const float a = ex2a(m[r] - mu), c = ex2a(mo - mu);
      l[r] = l[r] * a + lo2 * c;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[r][e] = acc[r][e] * a + __shfl_xor_sync(0xffffffffu, acc[r][e], x) * c;
      m[r] = mx;
    }
    if (sub == 0) {
#pragma unroll
      for (int e = 0; e < 8; ++e) s_acc[warp][r][d0 + e] = acc[r][e];
      if (lane == 0) { s_m[warp][r] = m[r]; s_l[warp][r] = l[r]; }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < R * HD; i += DC_WARPS * 32) {
    const int r = i / HD, d = i % HD;
    float mx = -INFINITY, ls = 0.f, v = 0.f;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) mx = fmaxf(mx, s_m[w][r]);
    const float mu = mx == -INFINITY ? 0.f : mx;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) {
      const float c = ex2a(s_m[w][r] - mu);
      ls += s_l[w][r] * c;
      v += s_acc[w][r][d] * c;
    }
    c_acc[r][d] = v;
    if (d == 0) { c_m[r] = mx; c_l[r] = ls; }
  }
  __syncthreads();
  cluster_sync_all();
  if (part == 0) {
    for (int i = threadIdx.x; i < rows * HD; i += DC_WARPS * 32) {
      const int r = i / HD, d = i % HD;
      float mx = -INFINITY, ls = 0.f, v = 0.f;
      for (int c = 0; c < parts; ++c) mx = fmaxf(mx, ld_cluster(&c_m[r], c));
      const float mu = mx == -INFINITY ? 0.f : mx;
      for (int c = 0; c < parts; ++c) {
        const float a = ex2a(ld_cluster(&c_m[r], c) - mu);
        ls += ld_cluster(&c_l[r], c) * a;
        v += ld_cluster(&c_acc[r][d], c) * a;
      }
      const int rep = r / p.Sq, iq = r % p.Sq;
      p.o[(((long long)b * p.Sq + iq) * p.Hq + h * n_rep + rep) * HD + d] = __float2bfloat16(ls > 0.f ? v / ls : 0.f);
    }
  }
  __syncthreads();
  cluster_sync_all();   // the first CTA has read the others' shared memory
}

template <int HD, int R>
int launch_decode(const DecodeParams& p, int parts, cudaStream_t stream) {
  const cudaError_t e = np_launch(decode_attn_kernel<HD, R>, dim3(parts, p.Hkv, p.B), DC_WARPS * 32, 0, stream, parts, p);
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

}  // namespace

// Called by np_gemm_bf16 for dense forward products of at most 64 rows where it is the faster one (few_rows_cost in
// gemm_sm100.cu); K must be a multiple of 8 and the
// rows of x and w 16-byte aligned.
int np_skinny_linear(const void* x, long long ldx, const void* w, long long ldw, int M, int N, int K, void* out, long long ldo,
                     int out_f32, float alpha, const float* bias, const void* cin, long long ldcin, cudaStream_t stream) {
  SkinnyParams p{};
  p.x = (const __nv_bfloat16*)x; p.w = (const __nv_bfloat16*)w; p.ldx = ldx; p.ldw = ldw;
  p.M = M; p.N = N; p.K = K; p.out = out; p.ldo = ldo; p.out_f32 = out_f32; p.alpha = alpha;
  p.bias = bias; p.cin = cin; p.ldcin = ldcin;
  const int grid = (N + 15) / 16;
  if (M <= 8) np_launch(skinny_linear_kernel<1, 4>, grid, SK_WARPS * 32, 0, stream, 1, p);
  else if (M <= 16) np_launch(skinny_linear_kernel<2, 4>, grid, SK_WARPS * 32, 0, stream, 1, p);
  else if (M <= 32) np_launch(skinny_linear_kernel<4, 2>, grid, SK_WARPS * 32, 0, stream, 1, p);
  else np_launch(skinny_linear_kernel<8, 2>, grid, SK_WARPS * 32, 0, stream, 1, p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 500 + (int)e;
}

NP_API int np_decode_attn(const NpDecodeArgs* a, void* stream) {
  if (a->B <= 0 || a->Sq <= 0 || a->past + a->fresh <= 0) return 0;
  if (a->Hkv <= 0 || a->Hq % a->Hkv || (a->head_dim != 64 && a->head_dim != 128)) return 1;
  const int rows = a->Hq / a->Hkv * a->Sq;
  if (rows > 8 || a->Hkv > 65535 || a->B > 65535) return 1;
  DecodeParams p{};
  p.q = (const __nv_bfloat16*)a->q; p.q_sb = a->q_sb; p.q_ss = a->q_ss; p.q_sh = a->q_sh;
  p.kc = (const __nv_bfloat16*)a->kc; p.kc_sb = a->kc_sb; p.kc_ss = a->kc_ss; p.kc_sh = a->kc_sh;
  p.vc = (const __nv_bfloat16*)a->vc; p.vc_sb = a->vc_sb; p.vc_ss = a->vc_ss; p.vc_sh = a->vc_sh;
  p.kn = (const __nv_bfloat16*)a->kn; p.kn_sb = a->kn_sb; p.kn_ss = a->kn_ss; p.kn_sh = a->kn_sh;
  p.vn = (const __nv_bfloat16*)a->vn; p.vn_sb = a->vn_sb; p.vn_ss = a->vn_ss; p.vn_sh = a->vn_sh;
  p.ko = (__nv_bfloat16*)a->ko; p.vo = (__nv_bfloat16*)a->vo; p.o = (__nv_bfloat16*)a->o;
  p.B = a->B; p.Sq = a->Sq; p.Hq = a->Hq; p.Hkv = a->Hkv; p.past = a->past; p.fresh = a->fresh; p.causal = a->causal;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  // enough CTAs for one and a half per SM (two fit), but no part below 64 keys, where the merge would outweigh the keys
  int parts = 1;
  while (parts < 8 && (long long)a->B * a->Hkv * parts < 222 && (a->past + a->fresh) / (2 * parts) >= 64) parts *= 2;
  cudaStream_t st = (cudaStream_t)stream;
  if (a->head_dim == 128) {
    if (rows <= 1) return launch_decode<128, 1>(p, parts, st);
    if (rows <= 2) return launch_decode<128, 2>(p, parts, st);
    if (rows <= 4) return launch_decode<128, 4>(p, parts, st);
    return launch_decode<128, 8>(p, parts, st);
  }
  if (rows <= 1) return launch_decode<64, 1>(p, parts, st);
  if (rows <= 2) return launch_decode<64, 2>(p, parts, st);
  if (rows <= 4) return launch_decode<64, 4>(p, parts, st);
  return launch_decode<64, 8>(p, parts, st);
}
