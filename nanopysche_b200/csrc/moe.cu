// MoE routing and expert-parallel token movement for sm_100a.
//
//  router_logits / router_topk / router_bwd : fp32 gate, DeepSeek-V3 score bias, top-k with softmax-
//      over-top-k or sigmoid+renorm gating, per-expert histogram, sum of full-softmax probabilities
//      and sum of logsumexp^2 (aux / z loss) in one pass; analytic backward to the logits.
//  capacity_plan : position of every token inside each expert it picked (index order), whole-token
//      drop beyond the capacity, positions among the kept tokens - no host sync.
//  ep_dispatch   : the all-to-all dispatch as peer stores: every kept (token, k) row is written
//      straight into the owning rank's expert-major receive buffer (region [local expert][source
//      rank], fixed size), optionally scaled (backward) or quantised to e4m3 with 1x128 scales
//      (FP8-Flow-MoE), together with the per-block row counts and per-row return addresses the
//      consuming grouped GEMM needs; the last CTA releases an epoch flag on every peer.
//  ep_combine    : waits (bounded) for the peers' epoch flags and reduces the K returned rows of each
//      token with the router weights, adding optional dense/shared/router-gradient terms.
//
// Replaces model/moe.py:133-321 (router), :1395-1448 (capacity), :360-498 (NCCL dispatcher: 4
// collectives + 3 host syncs per layer) and :1386-1390,1691-1714 (scatter-back) of the reference.
#include "common.cuh"
#include "args.h"

namespace {

constexpr int KID_DISPATCH = 10;
constexpr int KID_COMBINE = 11;
constexpr int MAX_E = 64;
constexpr int MAX_K = 8;

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  float2 a = np::unpack_bf16(u.x), b = np::unpack_bf16(u.y), c = np::unpack_bf16(u.z), d = np::unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(np::pack_bf16(f[0], f[1]), np::pack_bf16(f[2], f[3]), np::pack_bf16(f[4], f[5]),
                    np::pack_bf16(f[6], f[7]));
}

// ------------------------------------------------------------------ router
// logits[t, e] = <x[t], Wg[e]> + bias[e]  (fp32 accumulate, fp32 gate weights). Four warps share TOK tokens, each over the whole
// rows for EPW experts of a pass; MINB: CTAs per SM that the register count is held to, U: steps whose loads are in flight
// together. Bound by L1: the gate rows are 64 KB per TOK tokens at d 2048 and 8 experts, and each warp reads the tokens again. A
// warp to a token had the chain of its loads to wait for. 8 experts, us, before / now: 64 x 2048 7.2 / 3.5, 1024 10.8 / 5.0, 4096
// 20.7 / 13.3, 16384 41.4 / 40.6; 64 experts, 4096 x 1024 82 / 43. A quarter of the row to a warp, added over the warps, takes 11.7
// at 4096 and 30.3 at 16384, but forms the sums in another order; gate weights that differ in their last bits move the bf16 rows
// that they scale.
// Every token's sum is formed in the same order in all forms: a lane's vectors one after the other, then over the lanes.
template <int TOK, int EPW, int MINB, int U>
__global__ void __launch_bounds__(256, MINB) router_logits_kernel(const __nv_bfloat16* x, const float* wg, const float* bias,
                                                                  float* __restrict__ logits, int T, int D, int E,
                                                                  int* __restrict__ zero, int n_zero) {
  constexpr int PARTS = 4, V = TOK * EPW;   // V sums per warp, a power of two and at most one per lane
  np::pdl_begin();
  // what the kernel behind this one adds to (a fill of its own is a launch)
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n_zero; i += blockDim.x) zero[i] = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int tb = blockIdx.x * 2 * TOK; tb < T; tb += gridDim.x * 2 * TOK) {
    const int t0 = tb + warp / PARTS * TOK;
    for (int e0 = warp % PARTS * EPW; e0 < E; e0 += PARTS * EPW) {
      float acc[V];
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = 0.f;
#pragma unroll U
      for (int d = lane * 8; d < D; d += 256) {
        float xv[TOK][8];
#pragma unroll
        for (int k = 0; k < TOK; ++k) {
          if (t0 + k < T) {
            load8(x + (size_t)(t0 + k) * D + d, xv[k]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) xv[k][j] = 0.f;
          }
        }
#pragma unroll
        for (int e = 0; e < EPW; ++e) {
          if (e0 + e < E) {
            const float* wp = wg + (size_t)(e0 + e) * D + d;
            const float4 w0 = *reinterpret_cast<const float4*>(wp);
            const float4 w1 = *reinterpret_cast<const float4*>(wp + 4);
#pragma unroll
            for (int k = 0; k < TOK; ++k)
              acc[k * EPW + e] += xv[k][0] * w0.x + xv[k][1] * w0.y + xv[k][2] * w0.z + xv[k][3] * w0.w + xv[k][4] * w1.x +
                                  xv[k][5] * w1.y + xv[k][6] * w1.z + xv[k][7] * w1.w;
          }
        }
      }
      // sums over the lanes: each step hands half of the sums to the partner, until a lane has one of them
      int left = V;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if (left > 1) {
          left /= 2;
#pragma unroll
          for (int i = 0; i < V / 2; ++i) {
            if (i >= left) break;
            const float mine = lane & o ? acc[i + left] : acc[i], theirs = lane & o ? acc[i] : acc[i + left];
            acc[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
          }
        } else {
          acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        }
      }
      const int i = lane / (32 / V), t = t0 + i / EPW, e = e0 + i % EPW;
      if (lane % (32 / V) == 0 && t < T && e < E) logits[(size_t)t * E + e] = acc[0] + (bias ? bias[e] : 0.f);
    }
  }
}

// One thread per token. gating: 0 softmax over the selected logits, 1 sigmoid + renormalise.
// stats: counts[E] (int), psum[E] (sum of full-softmax probabilities), zsum[1] (sum of lse^2).
template <int EMAX>
__global__ void __launch_bounds__(256) router_topk_kernel(const float* logits,
                                                          const float* score_bias,
                                                          float* __restrict__ weights, int* __restrict__ indices,
                                                          int* __restrict__ counts, float* __restrict__ psum,
                                                          float* __restrict__ zsum, int T, int E, int K,
                                                          int gating) {
  np::pdl_begin();
  __shared__ int s_cnt[MAX_E];
  __shared__ float s_p[MAX_E];
  __shared__ float s_z;
  for (int i = threadIdx.x; i < E; i += blockDim.x) { s_cnt[i] = 0; s_p[i] = 0.f; }
  if (threadIdx.x == 0) s_z = 0.f;
  __syncthreads();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  // per-thread contributions to the statistics; reduced over the warp before they touch shared memory
  float pe[EMAX];
  float pz = 0.f;
  unsigned long long picked = 0ull;
#pragma unroll
  for (int e = 0; e < EMAX; ++e) pe[e] = 0.f;
  if (t < T) {
    float l[EMAX];  // EMAX is a compile-time bound so the logits stay in registers
    float mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < EMAX; ++e) {
      if (e >= E) { l[e] = -INFINITY; continue; }
      l[e] = logits[(size_t)t * E + e] + (score_bias ? score_bias[e] : 0.f);
      mx = fmaxf(mx, l[e]);
    }
    float se = 0.f;
#pragma unroll
    for (int e = 0; e < EMAX; ++e) se += (e < E) ? __expf(l[e] - mx) : 0.f;
    const float lse = mx + logf(se);
    pz = lse * lse;
#pragma unroll
    for (int e = 0; e < EMAX; ++e) pe[e] = (e < E) ? __expf(l[e] - lse) : 0.f;
    // top-k by repeated argmax (ties -> lowest index, as torch.topk on distinct values)
    int sel[MAX_K];
    float sv[MAX_K];
    unsigned long long used = 0ull;
    for (int k = 0; k < K; ++k) {
      int best = -1;
      float bv = -INFINITY;
#pragma unroll
      for (int e = 0; e < EMAX; ++e) {
        if (e >= E) continue;
        const float v = gating == 1 ? 1.f / (1.f + __expf(-l[e])) : l[e];
        if (!((used >> e) & 1ull) && (best < 0 || v > bv)) { best = e; bv = v; }
      }
      used |= 1ull << best;
      sel[k] = best;
      sv[k] = bv;
    }
    picked = used;
    float den = 0.f;
    if (gating == 1) {
      for (int k = 0; k < K; ++k) den += sv[k];
      den += 1e-8f;
      for (int k = 0; k < K; ++k) sv[k] /= den;
    } else {
      const float m0 = sv[0];  // the first pick is the largest selected logit
      for (int k = 0; k < K; ++k) { sv[k] = __expf(sv[k] - m0); den += sv[k]; }
      for (int k = 0; k < K; ++k) sv[k] /= den;
    }
    for (int k = 0; k < K; ++k) {
      weights[(size_t)t * K + k] = sv[k];
      indices[(size_t)t * K + k] = sel[k];
    }
  }
  {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int e = 0; e < EMAX; ++e) {
      if (e >= E) break;
      const float ps = np::warp_sum(pe[e]);
      const int c = __popc(__ballot_sync(0xffffffffu, (picked >> e) & 1ull));
      if (lane == 0) {
        atomicAdd(&s_p[e], ps);
        if (c) atomicAdd(&s_cnt[e], c);
      }
    }
    pz = np::warp_sum(pz);
    if (lane == 0) atomicAdd(&s_z, pz);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    if (s_cnt[i]) atomicAdd(&counts[i], s_cnt[i]);
    atomicAdd(&psum[i], s_p[i]);
  }
  if (threadIdx.x == 0) atomicAdd(zsum, s_z);
}

// f[e] = counts[e] / T and aux = E * sum_e f[e] * psum[e] / T + coef_z * zsum / T (one warp); NaN without tokens, the mean of
// nothing
__global__ void __launch_bounds__(32) router_aux_kernel(const int* counts, const float* psum,
                                                        const float* zsum, float coef_z, float* __restrict__ f,
                                                        float* __restrict__ aux, int T, int E) {
  np::pdl_begin();
  float s = 0.f;
  for (int e = threadIdx.x; e < E; e += 32) {
    const float fe = (float)counts[e] / (float)T;
    f[e] = fe;
    s += fe * (psum[e] / (float)T);
  }
  s = np::warp_sum(s);
  if (threadIdx.x == 0) aux[0] = (float)E * s + (coef_z != 0.f ? coef_z * zsum[0] / (float)T : 0.f);
}

// dlogits[t, :] from d(weights) and d(aux): aux = coef_lb * E * sum_i f_i * mean_t p[t,i]
//                                                + coef_z * mean_t lse_t^2
// f (fractions, [E]) is treated as a constant, as autograd does for the reference's one_hot count. EMAX bounds E at compile time so
// that a token's logits and gradients stay in registers (in local memory: 9.4 us at 4096 tokens and 8 experts).
template <int EMAX>
__global__ void __launch_bounds__(128) router_bwd_kernel(const float* logits,
                                                         const float* score_bias,
                                                         const float* weights,
                                                         const int* indices,
                                                         const float* dweights,
                                                         const float* f,
                                                         const float* daux, float coef_lb,
                                                         float coef_z, float* __restrict__ dlogits, int T, int E,
                                                         int K, int gating) {
  np::pdl_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  float l[EMAX], dl[EMAX];
  float mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < EMAX; ++e) {
    l[e] = e < E ? logits[(size_t)t * E + e] + (score_bias ? score_bias[e] : 0.f) : -INFINITY;
    mx = fmaxf(mx, l[e]);
    dl[e] = 0.f;
  }
  float se = 0.f;
#pragma unroll
  for (int e = 0; e < EMAX; ++e) se += e < E ? __expf(l[e] - mx) : 0.f;
  const float lse = mx + logf(se);
  const float da = daux ? daux[0] : 0.f;
  if (da != 0.f) {
    float fp = 0.f;
#pragma unroll
    for (int e = 0; e < EMAX; ++e)
      if (e < E) fp = fmaf(f[e], __expf(l[e] - lse), fp);
#pragma unroll
    for (int e = 0; e < EMAX; ++e) {
      if (e >= E) break;
      const float p = __expf(l[e] - lse);
      dl[e] += da * (coef_lb * (float)E / (float)T * p * (f[e] - fp) + coef_z * 2.f * lse / (float)T * p);
    }
  }
  if (dweights) {
    auto logit = [&](int e) {   // by selection: a variable index would put the array into local memory
      float v = l[0];
#pragma unroll
      for (int i = 1; i < EMAX; ++i) v = e == i ? l[i] : v;
      return v;
    };
    float wsum = 0.f, ssum = 1e-8f;
    for (int k = 0; k < K; ++k) {
      wsum += weights[(size_t)t * K + k] * dweights[(size_t)t * K + k];
      if (gating == 1) ssum += 1.f / (1.f + __expf(-logit(indices[(size_t)t * K + k])));
    }
    for (int k = 0; k < K; ++k) {
      const int e = indices[(size_t)t * K + k];
      const float w = weights[(size_t)t * K + k], dw = dweights[(size_t)t * K + k];
      float u = w, v = dw - wsum;   // u * v is added in one rounding
      if (gating != 0) {
        // w_k = s_k / (sum s + eps); ds_k = (dw_k - sum_j w_j dw_j) / (sum s + eps); dl = ds * s(1-s)
        const float s = 1.f / (1.f + __expf(-logit(e)));
        u = (dw - wsum) / ssum * s;
        v = 1.f - s;
      }
#pragma unroll
      for (int i = 0; i < EMAX; ++i) dl[i] = e == i ? fmaf(u, v, dl[i]) : dl[i];
    }
  }
#pragma unroll
  for (int e = 0; e < EMAX; ++e)
    if (e < E) dlogits[(size_t)t * E + e] = dl[e];
}

// partial[c, e, d] = sum over a chunk of 64 tokens of dl[t, e] * x[t, d] for EB experts a CTA. CTA = CT column threads (8 columns
// each) x 4 token lanes; a lane walks every fourth token of the chunk with U row loads in flight, the lanes are summed through
// shared memory. Beside them the first sums of the column sums of dl (the bias gradient): virtual thread (g, e) of 1024 / E groups
// adds rows g, g + groups, ... in four sums, into bias_part[g, e]. Bound by the chain of a lane's 16 tokens: a small batch takes
// narrow CTAs. us with the sum over the chunks, wide CTAs and the bias gradient in a launch of its own / chunks of 16 tokens
// (another order of the sums) / now: 64 x 2048, 8 experts 10.9 / 4.2 / 6.5, 512 x 768 10.6 / 5.6 / 6.7, 1000 x 1024, 16 19.6 / 11.0
// / 7.8, 4096 x 2048, 8 18.0 / 13.8 / 12.1.
constexpr int DG_TOK = 64, DG_BIAS = 1024;
template <int EB, int CT, int U>
__global__ void __launch_bounds__(CT * 4) router_dgate_kernel(const float* dl, const __nv_bfloat16* x, float* __restrict__ partial,
                                                              float* __restrict__ bias_part, int T, int D, int E) {
  np::pdl_begin();
  __shared__ float red[2][CT][EB * 8 + 1];
  __shared__ float s_dl[DG_TOK][EB];
  const int c = blockIdx.y, e0 = blockIdx.z * EB;
  const int t0 = c * DG_TOK, t1 = min(T, t0 + DG_TOK);
  const int tx = threadIdx.x % CT, ty = threadIdx.x / CT;
  const int d = (blockIdx.x * CT + tx) * 8;
  const bool col_ok = d < D;
  uint4 q[U];
  auto load = [&](int tb) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      q[u] = col_ok && tb + 4 * u < t1 ? *reinterpret_cast<const uint4*>(x + (size_t)(tb + 4 * u) * D + d) : make_uint4(0, 0, 0, 0);
  };
  load(t0 + ty);
  for (int i = threadIdx.x; i < (t1 - t0) * EB; i += CT * 4) {
    const int e = e0 + i % EB;
    s_dl[i / EB][i % EB] = e < E ? dl[(size_t)(t0 + i / EB) * E + e] : 0.f;
  }
  const int groups = DG_BIAS / E, ctas = gridDim.x * gridDim.y * gridDim.z;
  for (int v = ((blockIdx.z * gridDim.y + c) * gridDim.x + blockIdx.x) * CT * 4 + threadIdx.x; v < groups * E; v += ctas * CT * 4) {
    const int e = v % E;
    float a4[4] = {0.f, 0.f, 0.f, 0.f};
    int r = v / E;
    for (; r + 3 * groups < T; r += 4 * groups) {
#pragma unroll
      for (int u = 0; u < 4; ++u) a4[u] += dl[(size_t)(r + u * groups) * E + e];
    }
    for (; r < T; r += groups) a4[0] += dl[(size_t)r * E + e];
    bias_part[v] = (a4[0] + a4[1]) + (a4[2] + a4[3]);
  }
  __syncthreads();
  float acc[EB][8];
#pragma unroll
  for (int e = 0; e < EB; ++e)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[e][j] = 0.f;
  for (int tb = t0 + ty; tb < t1; tb += 4 * U) {   // tokens tb, tb + 4, ...
    if (tb != t0 + ty) load(tb);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (tb + 4 * u >= t1) break;
      float2 a = np::unpack_bf16(q[u].x), b = np::unpack_bf16(q[u].y), cc = np::unpack_bf16(q[u].z), dd = np::unpack_bf16(q[u].w);
      const float xv[8] = {a.x, a.y, b.x, b.y, cc.x, cc.y, dd.x, dd.y};
#pragma unroll
      for (int e = 0; e < EB; ++e) {
        const float g = s_dl[tb + 4 * u - t0][e];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[e][j] += g * xv[j];
      }
    }
  }
  if (ty >= 2) {   // lanes 2, 3 -> lanes 0, 1
#pragma unroll
    for (int e = 0; e < EB; ++e)
#pragma unroll
      for (int j = 0; j < 8; ++j) red[ty - 2][tx][e * 8 + j] = acc[e][j];
  }
  __syncthreads();
  if (ty < 2) {
#pragma unroll
    for (int e = 0; e < EB; ++e)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[e][j] += red[ty][tx][e * 8 + j];
  }
  __syncthreads();
  if (ty == 1) {   // lane 1 -> lane 0
#pragma unroll
    for (int e = 0; e < EB; ++e)
#pragma unroll
      for (int j = 0; j < 8; ++j) red[0][tx][e * 8 + j] = acc[e][j];
  }
  __syncthreads();
  if (ty == 0 && col_ok) {
#pragma unroll
    for (int e = 0; e < EB; ++e) {
      if (e0 + e < E) {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[e][j] += red[0][tx][e * 8 + j];
        float* dst = partial + ((size_t)c * E + e0 + e) * D + d;
        *reinterpret_cast<float4*>(dst) = make_float4(acc[e][0], acc[e][1], acc[e][2], acc[e][3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[e][4], acc[e][5], acc[e][6], acc[e][7]);
      }
    }
  }
}

// dx[t, :] = sum_e dl[t, e] * Wg[e, :] in bf16: the router's contribution to the gradient of its input (a
// [T, E] x [E, D] product with E of 8 to 64: one thread per 8 output columns, the gate rows come from L1).
__global__ void __launch_bounds__(256) router_dx_kernel(const float* dl, const float* wg,
                                                        __nv_bfloat16* __restrict__ dx, int T, int D, int E) {
  np::pdl_begin();
  const int vec_per_row = D >> 3;
  const long long total = (long long)T * vec_per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / vec_per_row), d = (int)(i % vec_per_row) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int e = 0; e < E; ++e) {
      const float g = dl[(size_t)t * E + e];
      const float4 w0 = *reinterpret_cast<const float4*>(wg + (size_t)e * D + d);
      const float4 w1 = *reinterpret_cast<const float4*>(wg + (size_t)e * D + d + 4);
      acc[0] += g * w0.x; acc[1] += g * w0.y; acc[2] += g * w0.z; acc[3] += g * w0.w;
      acc[4] += g * w1.x; acc[5] += g * w1.y; acc[6] += g * w1.z; acc[7] += g * w1.w;
    }
    *reinterpret_cast<uint4*>(dx + (size_t)t * D + d) = pack8(acc);
  }
}

// Same product for E <= 8 with D = 8 * blockDim.x: a thread keeps its 8 columns of all gate rows in registers and
// walks TOK tokens, so the only memory traffic per token is the [E] gradient row (broadcast) and one 16-byte store. The gradient
// rows of two tokens are loaded ahead: the first ones before the gate rows, the next ones before the last ones are used.
template <int TOK>
__global__ void __launch_bounds__(256, 2) router_dx_reg_kernel(const float* dl, const float* wg,
                                                            __nv_bfloat16* __restrict__ dx, int T, int D, int E) {
  np::pdl_begin();
  constexpr int G = 2;
  static_assert(TOK % G == 0, "whole groups");
  const int d = threadIdx.x * 8, t0 = blockIdx.x * TOK;
  float g[2][G][8], w[8][8];
  auto load_g = [&](int c) {
#pragma unroll
    for (int u = 0; u < G; ++u)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int t = t0 + c * G + u;
        g[c & 1][u][e] = t < T && e < E ? dl[(size_t)t * E + e] : 0.f;
      }
  };
  load_g(0);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float4 w0 = make_float4(0.f, 0.f, 0.f, 0.f), w1 = w0;
    if (e < E) {
      w0 = *reinterpret_cast<const float4*>(wg + (size_t)e * D + d);
      w1 = *reinterpret_cast<const float4*>(wg + (size_t)e * D + d + 4);
    }
    w[e][0] = w0.x; w[e][1] = w0.y; w[e][2] = w0.z; w[e][3] = w0.w;
    w[e][4] = w1.x; w[e][5] = w1.y; w[e][6] = w1.z; w[e][7] = w1.w;
  }
#pragma unroll
  for (int c = 0; c < TOK / G; ++c) {
    if (c + 1 < TOK / G) load_g(c + 1);
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int t = t0 + c * G + u;
      if (t >= T) break;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += g[c & 1][u][e] * w[e][j];
      *reinterpret_cast<uint4*>(dx + (size_t)t * D + d) = pack8(acc);
    }
  }
}

// out[c] (+)= column sums of `parts` rows of `cols` floats, 64 columns a CTA; the CTA behind the last adds up the bias gradient:
// bias_out[e] (+)= bias_part[0 .. groups, e] one after the other
__global__ void __launch_bounds__(64) router_dgate_sum_kernel(const float* partial, float* __restrict__ out, int parts, long long cols,
                                                              const float* bias_part, float* __restrict__ bias_out, int E, int accumulate) {
  np::pdl_begin();
  if (blockIdx.x * 64ll >= cols) {
    __shared__ float s_part[DG_BIAS];
    const int groups = DG_BIAS / E;
    for (int i = threadIdx.x; i < groups * E; i += 64) s_part[i] = bias_part[i];
    __syncthreads();
    if ((int)threadIdx.x < E) {
      float s = 0.f;
#pragma unroll 8
      for (int g = 0; g < groups; ++g) s += s_part[g * E + threadIdx.x];
      bias_out[threadIdx.x] = accumulate ? bias_out[threadIdx.x] + s : s;
    }
    return;
  }
  const long long c = blockIdx.x * 64ll + threadIdx.x;
  if (c >= cols) return;
  float a8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int p = 0;
  for (; p + 7 < parts; p += 8) {   // eight independent loads in flight
#pragma unroll
    for (int u = 0; u < 8; ++u) a8[u] += partial[(size_t)(p + u) * cols + c];
  }
  for (; p < parts; ++p) a8[0] += partial[(size_t)p * cols + c];
  const float s = ((a8[0] + a8[1]) + (a8[2] + a8[3])) + ((a8[4] + a8[5]) + (a8[6] + a8[7]));
  out[c] = accumulate ? out[c] + s : s;
}

// ------------------------------------------------------------------ capacity / positions
// One CTA of 32 warps, each over a contiguous run of slots (t, k), 32 at a time, a lane per slot. One ballot per bit of the expert
// number gives a lane the slots that picked the same expert as its own (its rank among them), and lane e those of expert e (and e +
// 32), so that the counters of up to 64 experts stand in two registers of a warp; more experts take further passes. Two passes over
// the slots with the warps' counts exchanged in between give the positions in token order. Phase 0 ranks every pick among all
// tokens that picked the expert and clears the flag of a token any of whose picks lies at or beyond `capacity` (capacity < 0: keep
// all); phase 1 ranks among the kept tokens. Up to 8192 slots stay in registers, more are read again (from L1). Bound by its chain
// of barriers and shuffles, one SM. A thread per run of tokens that scanned packed counters, us, before / now: 512 tokens, 8
// experts, top 2 7.5 / 4.3, 4096 18.5 / 9.3, 16384, 64, top 6 977 / 227.
// Outputs: slot_pos[t,k] (position among kept for expert idx[t,k], -1 if dropped), keep[T], counts_kept[E], drops[E] (tokens beyond
// capacity per expert), n_dropped[1].
constexpr int PLAN_CHUNKS = 8;     // runs of 32 slots that a warp holds at once
template <int EP>                  // experts per pass, 32 or 64
__global__ void __launch_bounds__(1024) capacity_plan_kernel(const int* indices, int T, int E, int K, int capacity,
                                                             int* __restrict__ slot_pos, int* keep, int* counts_kept,
                                                             int* __restrict__ drops, int* __restrict__ n_dropped,
                                                             int smem_flags, int* __restrict__ sent, int n_ranks,
                                                             long long* __restrict__ stats) {
  np::pdl_begin();
  extern __shared__ unsigned char s_keep[];   // a byte per token where they fit, else `keep` itself
  __shared__ int s_count[32][EP + 1], s_total[EP];
  __shared__ int s_dropped;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const long long n = (long long)T * K;
  const int chunks = (int)((n + 1023) / 1024);   // of a warp
  const bool held = chunks <= PLAN_CHUNKS;
  const long long s0 = (long long)warp * chunks * 32;
  const int t0 = (int)(s0 / K);                  // token and pick of the warp's first slot
  const unsigned k0 = (unsigned)(s0 % K);
  const int shift = K & (K - 1) ? -1 : __ffs(K) - 1;
  int ex[PLAN_CHUNKS], pos[PLAN_CHUNKS];
  auto slot = [&](int c) { return s0 + c * 32 + lane; };
  auto token = [&](int c) {
    const unsigned i = k0 + c * 32u + lane;
    return t0 + (int)(shift >= 0 ? i >> shift : i / (unsigned)K);
  };
  auto load = [&](int c0) {
#pragma unroll
    for (int u = 0; u < PLAN_CHUNKS; ++u) ex[u] = c0 + u < chunks && slot(c0 + u) < n ? indices[slot(c0 + u)] : -1;
  };
  auto is_kept = [&](int t) { return smem_flags ? s_keep[t] != 0 : keep[t] != 0; };
  load(0);
  if (threadIdx.x == 0) s_dropped = 0;
  for (int t = threadIdx.x; t < T; t += 1024) {
    if (smem_flags) s_keep[t] = 1;
    else keep[t] = 1;
  }
  __syncthreads();
  for (int phase = capacity < 0 ? 1 : 0; phase < 2; ++phase) {
    for (int e0 = 0; e0 < E; e0 += EP) {
      const int n_e = min(EP, E - e0), bits = n_e > 1 ? 32 - __clz(n_e - 1) : 0;
      int run_lo = 0, run_hi = 0;   // lane e: picks of experts e and e + 32 by the slots so far
      unsigned valid = 0;           // a bit per chunk: a pick of an expert of this pass by a kept token
      // counts the picks of a chunk; the position of this lane's slot among those of its expert, given those before it
      auto visit = [&](int u, int c, bool rank) {
        const int e = ex[u] - e0;
        const bool ok = e >= 0 && e < n_e && (phase == 0 || is_kept(token(c)));
        unsigned same = __ballot_sync(0xffffffffu, ok), lo = same, hi = 0;
        if (ok) valid |= 1u << u;
#pragma unroll
        for (int b = 0; b < 5; ++b) {
          if (b < bits) {
            const unsigned bit = (e >> b) & 1, v = __ballot_sync(0xffffffffu, bit);
            same &= v ^ (bit - 1u);
            lo &= v ^ (((lane >> b) & 1u) - 1u);
          }
        }
        int before = rank ? __shfl_sync(0xffffffffu, run_lo, e & 31) : 0;
        if (EP > 32 && bits == 6) {
          const unsigned bit = (e >> 5) & 1, v = __ballot_sync(0xffffffffu, bit);
          same &= v ^ (bit - 1u);
          hi = lo & v;
          lo &= ~v;
          const int h = rank ? __shfl_sync(0xffffffffu, run_hi, e & 31) : 0;
          if (bit) before = h;
          run_hi += __popc(hi);
        }
        run_lo += __popc(lo);
        return before + __popc(same & below);
      };
      for (int c0 = 0; c0 < chunks; c0 += PLAN_CHUNKS) {
        if (!held) load(c0);
#pragma unroll
        for (int u = 0; u < PLAN_CHUNKS; ++u) {
          if (c0 + u >= chunks) continue;
          if (held) pos[u] = visit(u, c0 + u, true);
          else visit(u, c0 + u, false);
        }
      }
      s_count[warp][lane] = run_lo;
      if (EP > 32) s_count[warp][lane + 32] = run_hi;
      __syncthreads();
      for (int e = warp; e < n_e; e += 32) {   // the warps before each one, per expert
        const int x = s_count[lane][e];
        int sum = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += y;
        }
        s_count[lane][e] = sum - x;
        if (lane == 31) s_total[e] = sum;
      }
      __syncthreads();
      run_lo = s_count[warp][lane];
      if (EP > 32) run_hi = s_count[warp][lane + 32];
      for (int c0 = 0; c0 < chunks; c0 += PLAN_CHUNKS) {
        if (!held) {
          valid = 0;
          load(c0);
        }
#pragma unroll
        for (int u = 0; u < PLAN_CHUNKS; ++u) {
          if (c0 + u >= chunks) continue;
          const int e = ex[u] - e0;
          int at;
          if (held) {
            at = __shfl_sync(0xffffffffu, run_lo, e & 31);
            if (EP > 32) {
              const int h = __shfl_sync(0xffffffffu, run_hi, e & 31);
              if (e >= 32) at = h;
            }
            at += pos[u];
          } else {
            at = visit(u, c0 + u, true);
          }
          const bool ok = (valid >> u) & 1u;
          if (phase == 0) {
            if (ok && at >= capacity) {   // only ever written to 0
              if (smem_flags) s_keep[token(c0 + u)] = 0;
              else keep[token(c0 + u)] = 0;
            }
          } else if (e >= 0 && e < n_e) {
            slot_pos[slot(c0 + u)] = ok ? at : -1;
          }
        }
      }
      if ((int)threadIdx.x < n_e) {
        const int e = threadIdx.x, c = s_total[e];
        if (phase == 0) {
          drops[e0 + e] = c > capacity ? c - capacity : 0;
        } else {
          counts_kept[e0 + e] = c;
          if (capacity < 0) drops[e0 + e] = 0;
        }
      }
    }
    __syncthreads();   // the flags of phase 0 are complete before phase 1 reads them; counts_kept before `sent` is formed
  }
  int nd = 0;
  for (int t = threadIdx.x; t < T; t += 1024) {
    const bool k = is_kept(t);
    if (smem_flags) keep[t] = k;
    nd += !k;
  }
  nd = __reduce_add_sync(0xffffffffu, nd);
  if (lane == 0 && nd) atomicAdd(&s_dropped, nd);
  __syncthreads();
  if (threadIdx.x == 0) {
    n_dropped[0] = s_dropped;
    if (stats) {   // last step's drops, all drops, all tokens
      stats[0] = s_dropped;
      stats[1] += s_dropped;
      stats[2] += T;
    }
  }
  if (sent) {      // kept rows per expert-parallel rank
    const int per_rank = E / n_ranks;
    for (int r = threadIdx.x; r < n_ranks; r += 1024) {
      int rows = 0;
      for (int e = r * per_rank; e < (r + 1) * per_rank; ++e) rows += counts_kept[e];
      sent[r] = rows;
    }
  }
}

// ------------------------------------------------------------------ EP dispatch (peer stores)
struct DispatchParams {
  const __nv_bfloat16* x;      // [T, D] source rows
  const int* indices;          // [T, K] expert of each slot
  const int* slot_pos;         // [T, K] position inside (expert, this source) region, -1 = dropped
  const int* counts_kept;      // [E]
  const float* slot_scale;     // [T, K] optional multiplier (backward: router weight), nullptr = 1
  int T, K, D, E, E_local, n_ranks, my_rank;
  int region_rows;             // rows reserved per (local expert, source) region, multiple of 128
  int quant;                   // 0: bf16 rows, 1: e4m3 rows + fp32 1x128 scales
  void* const* peer_rows;      // [n_ranks] receive buffer (bf16 [rows, D] or uint8 [rows, D])
  float* const* peer_scales;   // [n_ranks] fp32 [rows, D/128] (quant only)
  long long* const* peer_row_dst;   // [n_ranks] per-row return address (source << 40 | slot), -1 = padding
  int* const* peer_mblk_rows;  // [n_ranks] valid rows of every 128-row block of the receive buffer
  int* const* peer_src_blocks; // [n_ranks] [n_ranks] number of non-empty blocks sent by each source
  int* const* peer_flags;      // [n_ranks] [n_ranks] arrival epoch per source
  int* done_ctr;               // local CTA counter (zero between launches)
  int epoch;
  int write_meta;              // 1: also write row_dst / mblk_rows / src_blocks (forward); 0: rows only
  const int* epoch_base;       // optional device counter added to `epoch`
  int* zero_ctr;               // [n_ranks] tile counters of the pushing GEMM behind this dispatch, set to zero; may be nullptr
};

// Order what was written before what follows: for peers, or on this GPU when it is the only rank. A system-wide fence takes some
// 3 us, and there were four of them one after the other.
__device__ __forceinline__ void rank_fence(int n_ranks) {
  if (n_ranks > 1) __threadfence_system();
  else __threadfence();
}

__global__ void __launch_bounds__(256) ep_dispatch_kernel(const DispatchParams p) {
  np::pdl_begin();
  if (p.zero_ctr && blockIdx.x == 0)
    for (int i = threadIdx.x; i < p.n_ranks; i += blockDim.x) p.zero_ctr[i] = 0;
  np::CommSpan span(p.n_ranks > 1);
  const int lane = threadIdx.x & 31;
  const int warp_g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int slots = p.T * p.K;
  const int pad_items = p.E * 128;
  for (int it = warp_g; it < slots + pad_items; it += nwarps) {
    int e, pos;
    bool is_pad = it >= slots;
    float sc = 1.f;
    const __nv_bfloat16* src = nullptr;
    long long ret = -1;
    if (!is_pad) {
      pos = p.slot_pos[it];
      e = p.indices[it];
      if (pos < 0) continue;
      NP_DBG_SKIP_UNLESS(e >= 0 && e < p.E, KID_DISPATCH, e)
      src = p.x + (size_t)(it / p.K) * p.D;
      if (p.slot_scale) sc = p.slot_scale[it];
      ret = ((long long)p.my_rank << 40) | (long long)it;
    } else {
      e = (it - slots) >> 7;
      const int cnt = p.counts_kept[e];
      pos = cnt + ((it - slots) & 127);
      if (pos >= ((cnt + 127) & ~127)) continue;
    }
    if (pos >= p.region_rows) {  // cannot happen when region_rows >= capacity; recorded, not stored
      if (lane == 0) np::report(NP_ERR_BOUNDS, KID_DISPATCH, pos);
      continue;
    }
    const int peer = e / p.E_local, le = e - peer * p.E_local;
    const size_t row = ((size_t)le * p.n_ranks + p.my_rank) * p.region_rows + pos;
    if (!p.quant) {
      uint4* dst = reinterpret_cast<uint4*>((__nv_bfloat16*)p.peer_rows[peer] + row * p.D);
      // four vectors of the row in flight per lane: one load per store had the row's latency eight times over
      const int nv = p.D >> 3;
      for (int v0 = lane; v0 < nv; v0 += 128) {
        uint4 u[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          u[q] = make_uint4(0, 0, 0, 0);
          if (!is_pad && v0 + 32 * q < nv) u[q] = *reinterpret_cast<const uint4*>(src + (v0 + 32 * q) * 8);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (v0 + 32 * q >= nv) break;
          if (p.slot_scale) {
            float f[8];
            const float2 a = np::unpack_bf16(u[q].x), b = np::unpack_bf16(u[q].y), c = np::unpack_bf16(u[q].z),
                         d = np::unpack_bf16(u[q].w);
            f[0] = a.x * sc; f[1] = a.y * sc; f[2] = b.x * sc; f[3] = b.y * sc;
            f[4] = c.x * sc; f[5] = c.y * sc; f[6] = d.x * sc; f[7] = d.y * sc;
            u[q] = pack8(f);
          }
          dst[v0 + 32 * q] = u[q];
        }
      }
    } else {
      // 16 lanes x 8 elements = one 128-element scale block; two blocks per warp iteration
      uint2* dst = reinterpret_cast<uint2*>((uint8_t*)p.peer_rows[peer] + row * p.D);
      float* sdst = p.peer_scales[peer] + row * (p.D >> 7);
      for (int v = lane; v < (p.D >> 3); v += 32) {
        float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (!is_pad) {
          load8(src + v * 8, f);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] *= sc;
        }
        float am = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(f[j]));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
        float scale, inv;
        int e2 = -127;
        if (p.quant == 2) {   // power-of-two scale (UE8M0): ceil(log2(am / 448))
          if (am > 0.f) {
            int ex;
            const float mant = frexpf(__fdiv_rn(am, 448.f), &ex);
            e2 = (mant == 0.5f) ? ex - 1 : ex;
            e2 = max(-127, min(127, e2));
          }
          inv = exp2f((float)-e2);
          scale = 0.f;
        } else {
          scale = fmaxf(am, 1e-12f) / 448.f;
          inv = 1.f / scale;
        }
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lo |= (uint32_t)__nv_cvt_float_to_fp8(f[j] * inv, __NV_SATFINITE, __NV_E4M3) << (8 * j);
          hi |= (uint32_t)__nv_cvt_float_to_fp8(f[4 + j] * inv, __NV_SATFINITE, __NV_E4M3) << (8 * j);
        }
        dst[v] = make_uint2(lo, hi);
        if ((lane & 15) == 0) {
          if (p.quant == 2) {
            // exponent byte, four times, in the 512-byte chunk layout the block-scaled MMA reads (gemm_mxfp8_sm100.cu)
            const int r = (int)(row & 127), kb = v >> 4, nkb = p.D >> 7;
            uint8_t* sfb = reinterpret_cast<uint8_t*>(p.peer_scales[peer]);
            *reinterpret_cast<uint32_t*>(sfb + ((row >> 7) * nkb + kb) * 512 + (r & 31) * 16 + (r >> 5) * 4) =
                (uint32_t)(e2 + 127) * 0x01010101u;
          } else {
            sdst[v >> 4] = scale;
          }
        }
      }
    }
    if (p.write_meta && lane == 0) p.peer_row_dst[peer][row] = ret;
  }
  // ---- completion: last CTA publishes the block table and releases the epoch flags
  rank_fence(p.n_ranks);
  __syncthreads();
  __shared__ int s_last;
  if (threadIdx.x == 0) s_last = (atomicAdd(p.done_ctr, 1) == (int)gridDim.x - 1);
  __syncthreads();
  if (!s_last) return;
  rank_fence(p.n_ranks);
  const int bpr = p.region_rows >> 7;  // blocks per region
  if (p.write_meta) {
    for (int i = threadIdx.x; i < p.E * bpr; i += blockDim.x) {
      const int e = i / bpr, b = i - e * bpr;
      const int peer = e / p.E_local, le = e - peer * p.E_local;
      int r = p.counts_kept[e] - b * 128;
      r = r < 0 ? 0 : (r > 128 ? 128 : r);
      // a block with any row is processed whole (its padding rows are zero)
      p.peer_mblk_rows[peer][((size_t)le * p.n_ranks + p.my_rank) * bpr + b] = r > 0 ? 128 : 0;
    }
    for (int peer = threadIdx.x; peer < p.n_ranks; peer += blockDim.x) {
      int nb = 0;
      for (int le = 0; le < p.E_local; ++le) nb += (p.counts_kept[peer * p.E_local + le] + 127) >> 7;
      p.peer_src_blocks[peer][p.my_rank] = nb;
    }
  }
  rank_fence(p.n_ranks);
  __syncthreads();
  const int epoch = p.epoch + (p.epoch_base ? *p.epoch_base : 0);
  if (p.n_ranks == 1) {
    if (threadIdx.x == 0) np::st_release_gpu(p.peer_flags[0], epoch);
  } else {
    for (int peer = threadIdx.x; peer < p.n_ranks; peer += blockDim.x) np::st_release_sys(p.peer_flags[peer] + p.my_rank, epoch);
  }
  if (threadIdx.x == 0) *p.done_ctr = 0;
}

// ------------------------------------------------------------------ EP combine (reduce at the source)
struct CombineParams {
  const __nv_bfloat16* rows;   // [T*K, D] rows returned by the experts (slot-major)
  const int* slot_pos;         // [T, K], -1 = dropped slot (contributes zero)
  const float* weights;        // [T, K] router weights, nullptr = 1 (backward)
  const __nv_bfloat16* add1;   // optional [T, D] term added to every token
  const __nv_bfloat16* add2;   // optional second [T, D] term
  const float* dl;             // optional router term: out += dl[t, :] @ wg   (dl [T, E], wg [E, D])
  const float* wg;
  __nv_bfloat16* out;          // [T, D]
  int T, K, D, E;
  const int* flags;            // [n_ranks] completion epoch written by each peer, nullptr = no wait
  const int* sent_to_peer;     // [n_ranks] rows this rank sent to each peer (0 = nothing to wait for)
  int n_ranks, epoch;
  unsigned long long limit_ns;
  const int* epoch_base;
};

__global__ void __launch_bounds__(256) ep_combine_kernel(const CombineParams p) {
  np::pdl_begin();
  __shared__ int s_ok;
  if (p.flags) {
    if (threadIdx.x == 0) s_ok = 1;
    __syncthreads();
    if ((int)threadIdx.x < p.n_ranks && p.sent_to_peer[threadIdx.x] > 0) {
      if (!np::wait_flag_ge(p.flags + threadIdx.x, p.epoch + (p.epoch_base ? *p.epoch_base : 0), p.limit_ns, KID_COMBINE,
                            threadIdx.x)) s_ok = 0;
    }
    __syncthreads();
    if (!s_ok) return;
  }
  const int vec_per_row = p.D >> 3;
  const long long total = (long long)p.T * vec_per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = total <= 0x7fffffff ? (int)((unsigned)i / (unsigned)vec_per_row) : (int)(i / vec_per_row);
    const int d = (int)(i - (long long)t * vec_per_row) * 8;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int k0 = 0; k0 < p.K; k0 += 2) {   // two rows in flight
      uint4 q[2];
      float w[2];
      bool on[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const size_t slot = (size_t)t * p.K + k0 + u;
        on[u] = k0 + u < p.K && p.slot_pos[slot] >= 0;
        q[u] = make_uint4(0, 0, 0, 0);
        w[u] = 0.f;
        if (on[u]) {
          on[u] = false;   // debug build: a position out of range is reported and its row left out
          NP_DBG_SKIP_UNLESS(p.slot_pos[slot] < (1 << 24), KID_COMBINE, p.slot_pos[slot])
          on[u] = true;
        }
        if (on[u]) {
          q[u] = *reinterpret_cast<const uint4*>(p.rows + slot * p.D + d);
          w[u] = p.weights ? p.weights[slot] : 1.f;
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (!on[u]) continue;
        const float2 a = np::unpack_bf16(q[u].x), b = np::unpack_bf16(q[u].y), c = np::unpack_bf16(q[u].z),
                     e = np::unpack_bf16(q[u].w);
        acc[0] += w[u] * a.x; acc[1] += w[u] * a.y; acc[2] += w[u] * b.x; acc[3] += w[u] * b.y;
        acc[4] += w[u] * c.x; acc[5] += w[u] * c.y; acc[6] += w[u] * e.x; acc[7] += w[u] * e.y;
      }
    }
    if (p.add1) {
      float f[8];
      load8(p.add1 + (size_t)t * p.D + d, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += f[j];
    }
    if (p.add2) {
      float f[8];
      load8(p.add2 + (size_t)t * p.D + d, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += f[j];
    }
    if (p.dl) {
      for (int e = 0; e < p.E; ++e) {
        const float g = p.dl[(size_t)t * p.E + e];
        const float4 w0 = *reinterpret_cast<const float4*>(p.wg + (size_t)e * p.D + d);
        const float4 w1 = *reinterpret_cast<const float4*>(p.wg + (size_t)e * p.D + d + 4);
        acc[0] += g * w0.x; acc[1] += g * w0.y; acc[2] += g * w0.z; acc[3] += g * w0.w;
        acc[4] += g * w1.x; acc[5] += g * w1.y; acc[6] += g * w1.z; acc[7] += g * w1.w;
      }
    }
    *reinterpret_cast<uint4*>(p.out + (size_t)t * p.D + d) = pack8(acc);
  }
}

// dots[t, k] = <a[t, :], rows[t*K + k, :]>  (0 for dropped slots); one warp per slot.
__global__ void __launch_bounds__(256) slot_dot_kernel(const __nv_bfloat16* a,
                                                       const __nv_bfloat16* rows,
                                                       const int* slot_pos, float* __restrict__ dots,
                                                       int T, int K, int D) {
  np::pdl_begin();
  const int lane = threadIdx.x & 31;
  const int warp_g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int s = warp_g; s < T * K; s += nwarps) {
    float acc = 0.f;
    if (slot_pos[s] >= 0) {
      const int t = s / K;
      for (int d = lane * 8; d < D; d += 256) {
        float f[8], g[8];
        load8(a + (size_t)t * D + d, f);
        load8(rows + (size_t)s * D + d, g);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc += f[j] * g[j];
      }
    }
    acc = np::warp_sum(acc);
    if (lane == 0) dots[s] = acc;
  }
}

}  // namespace

#define CHECK_LAUNCH() do { cudaError_t e_ = cudaGetLastError(); return e_ == cudaSuccess ? 0 : 500 + (int)e_; } while (0)

// zero [n_zero]: set to zero (n_zero may be 0)
NP_API int np_router_logits(const void* x, const float* wg, const float* bias, float* logits, int T, int D, int E, int* zero,
                            int n_zero, void* stream) {
  if (D % 8 || T <= 0) return T <= 0 ? 0 : 1;
  auto run = [&](auto kernel, int tok) {
    const int blocks = (T + 2 * tok - 1) / (2 * tok);
    np_launch(kernel, (unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, (cudaStream_t)stream, 1, (const __nv_bfloat16*)x, wg, bias,
              logits, T, D, E, zero, n_zero);
  };
  // Two tokens per four warps with two experts a warp and the vectors of four steps in flight as long as that is one wave of CTAs,
  // then four, which read the gate rows half as often: an expert a warp and four steps, from nine experts on four experts a warp,
  // which read the tokens a quarter as often. us, first / second / third: 64 x 2048, 8 experts 3.5 / 5.2 / 11.5, 1024 5.0 / 5.6 /
  // 11.8, 2048 8.4 / 7.6 / 11.9, 4096 14.7 / 13.3 / 19.1; 2472 x 1024, 16 experts 10.8 / 11.9 / 11.1; 4096 x 1024, 64 53 / 47 / 43.
  if (T <= 148 * 2 * 4) run(router_logits_kernel<2, 2, 2, 4>, 2);
  else if (E <= 8) run(router_logits_kernel<4, 1, 2, 4>, 4);
  else run(router_logits_kernel<4, 4, 2, 1>, 4);
  CHECK_LAUNCH();
}

// counts/psum/zsum must be zeroed by the caller before the launch.
NP_API int np_router_topk(const float* logits, const float* score_bias, float* weights, int* indices, int* counts,
                          float* psum, float* zsum, int T, int E, int K, int gating, void* stream) {
  if (E > MAX_E || K > MAX_K || K > E) return 1;
  if (T <= 0) return 0;
#define TOPK(EM) np_launch(router_topk_kernel<EM>, (T + 127) / 128, 128, 0, (cudaStream_t)stream, 1, \
      logits, score_bias, weights, indices, counts, psum, zsum, T, E, K, gating)
  if (E <= 8) TOPK(8);
  else if (E <= 16) TOPK(16);
  else if (E <= 32) TOPK(32);
  else TOPK(64);
#undef TOPK
  CHECK_LAUNCH();
}

NP_API int np_router_aux(const int* counts, const float* psum, const float* zsum, float coef_z, float* f, float* aux, int T,
                         int E, void* stream) {
  if (T < 0 || E > MAX_E) return 1;
  np_launch(router_aux_kernel, 1, 32, 0, (cudaStream_t)stream, 1, counts, psum, zsum, coef_z, f, aux, T, E);
  CHECK_LAUNCH();
}

NP_API int np_router_bwd(const float* logits, const float* score_bias, const float* weights, const int* indices,
                         const float* dweights, const float* f, const float* daux, float coef_lb, float coef_z,
                         float* dlogits, int T, int E, int K, int gating, void* stream) {
  if (E > MAX_E || K > MAX_K) return 1;
  if (T <= 0) return 0;
#define RBWD(EM) np_launch(router_bwd_kernel<EM>, (T + 127) / 128, 128, 0, (cudaStream_t)stream, 1, logits, score_bias, weights, \
      indices, dweights, f, daux, coef_lb, coef_z, dlogits, T, E, K, gating)
  if (E <= 8) RBWD(8);
  else if (E <= 16) RBWD(16);
  else if (E <= 32) RBWD(32);
  else RBWD(64);
#undef RBWD
  CHECK_LAUNCH();
}

// Floats of the scratch buffer of np_router_dgate
NP_API long long np_router_dgate_scratch(int T, int D, int E) { return (long long)((T + DG_TOK - 1) / DG_TOK) * E * D + DG_BIAS; }
// dwg[E, D] (+)= dl^T x ; dbias[E] (+)= column sums of dl.
NP_API int np_router_dgate(const float* dl, const void* x, float* dwg, float* dbias, float* scratch, int T, int D,
                           int E, int accumulate, void* stream) {
  if (D % 8 || E > MAX_E) return 1;
  if (T <= 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const int parts = (T + DG_TOK - 1) / DG_TOK;
  const long long n = (long long)E * D;
  float* bias_part = scratch + parts * n;
  auto run = [&](auto kernel, int ct) {
    np_launch(kernel, dim3((D / 8 + ct - 1) / ct, parts, (E + 7) / 8), ct * 4, 0, s, 1, dl, (const __nv_bfloat16*)x, scratch,
              bias_part, T, D, E);
  };
  if (T <= 1024) run(router_dgate_kernel<8, 16, 8>, 16);
  else run(router_dgate_kernel<8, 64, 4>, 64);
  np_launch(router_dgate_sum_kernel, (unsigned)((n + 63) / 64 + (dbias ? 1 : 0)), 64, 0, s, 1, scratch, dwg, parts, n, bias_part,
            dbias, E, accumulate);
  CHECK_LAUNCH();
}

NP_API int np_router_dx(const float* dl, const float* wg, void* dx, int T, int D, int E, void* stream) {
  if (D % 8) return 1;
  if (T <= 0) return 0;
  if (E <= 8 && D % 8 == 0 && D / 8 <= 256 && D / 8 >= 32) {
    constexpr int TOK = 8;
    np_launch(router_dx_reg_kernel<TOK>, (unsigned)((T + TOK - 1) / TOK), D / 8, 0, (cudaStream_t)stream, 1,
        dl, wg, (__nv_bfloat16*)dx, T, D, E);
    CHECK_LAUNCH();
  }
  const long long blocks = ((long long)T * (D / 8) + 255) / 256;
  np_launch(router_dx_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream, 1, dl, wg, (__nv_bfloat16*)dx, T, D, E);
  CHECK_LAUNCH();
}

// sent [n_ranks]: kept rows per rank (may be null); stats [3]: last dropped, total dropped, total tokens (may be null).
NP_API int np_capacity_plan(const int* indices, int T, int E, int K, int capacity, int* slot_pos, int* keep, int* counts_kept,
                            int* drops, int* n_dropped, int* sent, int n_ranks, long long* stats, void* stream) {
  if (K > MAX_K || (sent && (n_ranks <= 0 || E % n_ranks))) return 1;
  if (T <= 0) return 0;
  const int flags_fit = T <= 200 * 1024;   // a byte per token beside the counts of the warps
  static NpPerDeviceOnce attr_once;
  bool& attr_set = *attr_once.slot();
  if (flags_fit && !attr_set) {
    cudaError_t e = cudaFuncSetAttribute(capacity_plan_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(capacity_plan_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return 400 + (int)e;
    attr_set = true;
  }
  np_launch(E <= 32 ? capacity_plan_kernel<32> : capacity_plan_kernel<64>, 1, 1024, flags_fit ? (size_t)T : 0, (cudaStream_t)stream,
            1, indices, T, E, K, capacity, slot_pos, keep, counts_kept, drops, n_dropped, flags_fit, sent, n_ranks, stats);
  CHECK_LAUNCH();
}

// without either
NP_API int np_capacity_scan(const int* indices, int T, int E, int K, int capacity, int* slot_pos, int* keep, int* counts_kept,
                            int* drops, int* n_dropped, void* stream) {
  return np_capacity_plan(indices, T, E, K, capacity, slot_pos, keep, counts_kept, drops, n_dropped, nullptr, 0, nullptr, stream);
}

NP_API int np_ep_dispatch(const NpDispatchArgs* a, void* stream) {
  if (a->D % 128 || a->region_rows % 128 || a->E % a->E_local || (a->quant && a->D % 256)) return 1;
  DispatchParams p;
  p.x = (const __nv_bfloat16*)a->x; p.indices = a->indices; p.slot_pos = a->slot_pos; p.counts_kept = a->counts_kept;
  p.slot_scale = a->slot_scale; p.T = a->T; p.K = a->K; p.D = a->D; p.E = a->E; p.E_local = a->E_local;
  p.n_ranks = a->n_ranks; p.my_rank = a->my_rank; p.region_rows = a->region_rows; p.quant = a->quant;
  p.peer_rows = a->peer_rows; p.peer_scales = a->peer_scales; p.peer_row_dst = a->peer_row_dst;
  p.peer_mblk_rows = a->peer_mblk_rows; p.peer_src_blocks = a->peer_src_blocks; p.peer_flags = a->peer_flags;
  p.done_ctr = a->done_ctr; p.epoch = a->epoch; p.write_meta = a->write_meta;
  p.epoch_base = a->epoch_base; p.zero_ctr = a->zero_ctr;
  const int items = a->T * a->K + a->E * 128;
  int grid = (items + 7) / 8;
  const int cap = a->max_ctas > 0 ? a->max_ctas : 148 * 8;   // a row per warp as long as they fit the chip at once
  if (grid > cap) grid = cap;
  if (grid < 1) grid = 1;
  np_launch(ep_dispatch_kernel, grid, 256, 0, (cudaStream_t)stream, 1, p);
  CHECK_LAUNCH();
}

NP_API int np_ep_combine(const NpCombineArgs* a, void* stream) {
  if (a->D % 8 || a->n_ranks > 256) return 1;
  if (a->T <= 0) return 0;
  CombineParams p;
  p.rows = (const __nv_bfloat16*)a->rows; p.slot_pos = a->slot_pos; p.weights = a->weights;
  p.add1 = (const __nv_bfloat16*)a->add1; p.add2 = (const __nv_bfloat16*)a->add2; p.dl = a->dl; p.wg = a->wg;
  p.out = (__nv_bfloat16*)a->out; p.T = a->T; p.K = a->K; p.D = a->D; p.E = a->E; p.flags = a->flags;
  p.sent_to_peer = a->sent_to_peer; p.n_ranks = a->n_ranks; p.epoch = a->epoch;
  p.limit_ns = a->limit_ns ? a->limit_ns : NP_WAIT_LIMIT_NS;
  p.epoch_base = a->epoch_base;
  long long work = (long long)a->T * (a->D / 8);
  int grid = (int)((work + 255) / 256);
  if (grid > 148 * 8) grid = 148 * 8;
  np_launch(ep_combine_kernel, grid, 256, 0, (cudaStream_t)stream, 1, p);
  CHECK_LAUNCH();
}

NP_API int np_slot_dot(const void* a, const void* rows, const int* slot_pos, float* dots, int T, int K, int D,
                       void* stream) {
  if (D % 8) return 1;
  if (T <= 0) return 0;
  int grid = (T * K + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
  np_launch(slot_dot_kernel, grid, 256, 0, (cudaStream_t)stream, 1, (const __nv_bfloat16*)a, (const __nv_bfloat16*)rows, slot_pos,
                                                          dots, T, K, D);
  CHECK_LAUNCH();
}
