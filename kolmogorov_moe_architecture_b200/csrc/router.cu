// Routing decisions as single kernels (CUDA cores; the inputs are tiny next to the expert GEMMs, the
// point is one launch instead of a chain of softmax / top-k / sort / bincount launches, and no
// intermediate tensors).
//
//   route_topk      token-choice router tail: softmax over experts -> top-k -> renormalise, plus the
//                   load-balance and z-loss partial sums (sum of probabilities and assignment count
//                   per expert, sum of logsumexp^2).            reference: moe_arch/model/moe.py:441-460, 840-939
//   seq_topk        per-row top-k of a (rows, S) score matrix, one CTA per row, bitonic sort in shared
//                   memory.  mode 0 (mixture-of-depths): keep the k largest logits, emit their indices in
//                   ascending order and a softmax over the kept logits.  reference: moe_arch/model/mod.py:93-112
//                   mode 1 (expert choice): softmax over the whole row, keep the k largest probabilities
//                   in descending order, renormalise.          reference: moe_arch/model/moe.py:494-530
// Each has a backward kernel producing d(logits).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include "kmoe_api.h"
#include "ptx.cuh"

namespace kmoe {

constexpr int ROUTE_MAX_E = 128;
constexpr int ROUTE_MAX_K = 8;

// ---------------------------------------------------------------------------- token choice
// One warp per token, lane l holds experts l, l + 32, ... in registers; logits fp32 or bf16 (T, E).  The per-expert sums
// of probabilities and assignments are carried in the lanes that own the experts and meet once per CTA.  What bounds it is
// latency (a chain of 2 + k warp reductions per token), so the grid gives every SM many warps.  One thread per token, with
// the row's probabilities in local memory, took 13.1 us for 6144 x 16 and 53 us for 4096 x 64 (backward 5.7 and 20.3);
// this way 6.4 and 6.5 us (4.0 and 3.7).
constexpr int ROUTE_WARPS = 4;
constexpr int ROUTE_PER_LANE = ROUTE_MAX_E / 32;
__device__ __forceinline__ float route_in(const float* p) { return *p; }
__device__ __forceinline__ float route_in(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void route_out(float* p, float v) { *p = v; }
__device__ __forceinline__ void route_out(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

template <typename T_>
__global__ void __launch_bounds__(32 * ROUTE_WARPS)
route_topk_fwd_kernel(const T_* __restrict__ logits, int T, int E, int k, float* __restrict__ w_f32,
                      T_* __restrict__ w_out, long long* __restrict__ idx_out, float* __restrict__ lse_out,
                      float* __restrict__ p_sum, float* __restrict__ counts, float* __restrict__ z_sum) {
  __shared__ float s_p[ROUTE_WARPS][ROUTE_MAX_E], s_c[ROUTE_WARPS][ROUTE_MAX_E], s_z[ROUTE_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = gridDim.x * ROUTE_WARPS;
  float psum[ROUTE_PER_LANE], cnt[ROUTE_PER_LANE], z = 0.f;
#pragma unroll
  for (int i = 0; i < ROUTE_PER_LANE; ++i) psum[i] = cnt[i] = 0.f;
  for (int t = blockIdx.x * ROUTE_WARPS + warp; t < T; t += warps) {
    const T_* row = logits + (size_t)t * E;
    float x[ROUTE_PER_LANE];
    float mx = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < ROUTE_PER_LANE; ++i) {
      const int e = lane + 32 * i;
      x[i] = e < E ? route_in(row + e) : -CUDART_INF_F;
      mx = fmaxf(mx, x[i]);
    }
    mx = warp_max(mx);
    float den = 0.f;
#pragma unroll
    for (int i = 0; i < ROUTE_PER_LANE; ++i)
      if (lane + 32 * i < E) den += __expf(x[i] - mx);
    den = warp_sum(den);
    const float lse = mx + __logf(den), inv = 1.f / den;
    z += lse * lse;
    unsigned used = 0;                  // bit i: this lane's expert lane + 32 i is taken
    float pv[ROUTE_MAX_K], s = 0.f;
    int sel[ROUTE_MAX_K];
#pragma unroll
    for (int j = 0; j < ROUTE_MAX_K; ++j) {
      if (j >= k) break;
      float best = -CUDART_INF_F;
      int be = ROUTE_MAX_E;             // first maximum wins ties, like a stable arg-max; no candidate at all: expert 0
#pragma unroll
      for (int i = 0; i < ROUTE_PER_LANE; ++i)
        if (!(used >> i & 1) && x[i] > best) { best = x[i]; be = lane + 32 * i; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oe = __shfl_xor_sync(0xffffffffu, be, o);
        if (ob > best || (ob == best && oe < be)) { best = ob; be = oe; }
      }
      if (be >= E) be = 0;
#pragma unroll
      for (int i = 0; i < ROUTE_PER_LANE; ++i)
        if (be == lane + 32 * i) {
          used |= 1u << i;
          cnt[i] += 1.f;
        }
      sel[j] = be;
      pv[j] = __expf(best - mx) * inv;
      s += pv[j];
    }
#pragma unroll
    for (int j = 0; j < ROUTE_MAX_K; ++j) {
      if (j >= k) break;
      if (lane == j) {
        const float w = pv[j] / s;
        w_f32[(size_t)t * k + j] = w;
        if (w_out != nullptr) route_out(w_out + (size_t)t * k + j, w);
        idx_out[(size_t)t * k + j] = sel[j];
      }
    }
    if (lane == 0) lse_out[t] = lse;
#pragma unroll
    for (int i = 0; i < ROUTE_PER_LANE; ++i)
      if (lane + 32 * i < E) psum[i] += __expf(x[i] - mx) * inv;
  }
#pragma unroll
  for (int i = 0; i < ROUTE_PER_LANE; ++i) {
    s_p[warp][lane + 32 * i] = psum[i];
    s_c[warp][lane + 32 * i] = cnt[i];
  }
  if (lane == 0) s_z[warp] = z;
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += 32 * ROUTE_WARPS) {
    float a = 0.f, c = 0.f;
#pragma unroll
    for (int q = 0; q < ROUTE_WARPS; ++q) { a += s_p[q][e]; c += s_c[q][e]; }
    if (a != 0.f) atomicAdd(&p_sum[e], a);
    if (c != 0.f) atomicAdd(&counts[e], c);
  }
  if (threadIdx.x == 0) {
    float a = 0.f;
#pragma unroll
    for (int q = 0; q < ROUTE_WARPS; ++q) a += s_z[q];
    if (a != 0.f) atomicAdd(z_sum, a);
  }
}

// aux = c_lb * sum_e p_sum[e] counts[e] + c_z * z_sum   (one warp)
__global__ void route_aux_kernel(const float* __restrict__ acc, int E, float c_lb, float c_z, float* __restrict__ aux) {
  float v = 0.f;
  for (int e = threadIdx.x; e < E; e += 32) v += acc[e] * acc[E + e];
  v = warp_sum(v);
  if (threadIdx.x == 0) *aux = c_lb * v + c_z * acc[2 * E];
}

// dlogits = softmax-backward of [renorm-backward(dw) at the selected experts + c_lb[e]] + c_z * 2 lse p
//   c_lb[e] = d_aux * w_lb * E * f_e / T   (the assignment fractions f_e are constants, as in the reference)
//   c_z     = d_aux * w_z / T
template <typename T_>
__global__ void __launch_bounds__(32 * ROUTE_WARPS)
route_topk_bwd_kernel(const T_* __restrict__ logits, const float* __restrict__ lse, const long long* __restrict__ idx,
                      const float* __restrict__ w, const T_* __restrict__ dw, const float* __restrict__ counts,
                      const float* __restrict__ d_aux, float w_lb, float w_z, int T, int E, int k,
                      T_* __restrict__ dlogits) {
  const int lane = threadIdx.x & 31, warps = gridDim.x * ROUTE_WARPS;
  const float da = d_aux ? *d_aux : 0.f;
  const float lb_scale = da * w_lb * (float)E / ((float)T * (float)T * (float)k);
  float lb[ROUTE_PER_LANE];
#pragma unroll
  for (int i = 0; i < ROUTE_PER_LANE; ++i) lb[i] = lane + 32 * i < E ? lb_scale * counts[lane + 32 * i] : 0.f;
  for (int t = blockIdx.x * ROUTE_WARPS + (threadIdx.x >> 5); t < T; t += warps) {
    const T_* row = logits + (size_t)t * E;
    const float l = lse[t];
    float p[ROUTE_PER_LANE], dp[ROUTE_PER_LANE];
#pragma unroll
    for (int i = 0; i < ROUTE_PER_LANE; ++i) {
      const int e = lane + 32 * i;
      p[i] = e < E ? __expf(route_in(row + e) - l) : 0.f;
      dp[i] = lb[i];
    }
    // lane j < k holds assignment j
    const bool mine = lane < k;
    const int ej = mine ? (int)idx[(size_t)t * k + lane] : 0;
    const float dwj = (mine && dw != nullptr) ? route_in(dw + (size_t)t * k + lane) : 0.f;
    const float dot_w = warp_sum(mine ? dwj * w[(size_t)t * k + lane] : 0.f);
    float s = 0.f;                      // probability of the selected experts
    for (int j = 0; j < k; ++j) {
      const int e = __shfl_sync(0xffffffffu, ej, j);
      float pe = 0.f;
#pragma unroll
      for (int i = 0; i < ROUTE_PER_LANE; ++i)
        if (e >> 5 == i) pe = p[i];
      s += __shfl_sync(0xffffffffu, pe, e & 31);
    }
    for (int j = 0; j < k; ++j) {
      const int e = __shfl_sync(0xffffffffu, ej, j);
      const float g = (__shfl_sync(0xffffffffu, dwj, j) - dot_w) / s;
#pragma unroll
      for (int i = 0; i < ROUTE_PER_LANE; ++i)
        if (e == lane + 32 * i) dp[i] += g;
    }
    float pd = 0.f;
#pragma unroll
    for (int i = 0; i < ROUTE_PER_LANE; ++i) pd += p[i] * dp[i];
    pd = warp_sum(pd);
    const float cz = da * w_z * 2.f * l / (float)T;
#pragma unroll
    for (int i = 0; i < ROUTE_PER_LANE; ++i)
      if (lane + 32 * i < E) route_out(dlogits + (size_t)t * E + lane + 32 * i, p[i] * (dp[i] - pd) + cz * p[i]);
  }
}

// ---------------------------------------------------------------------------- per-row top-k
// Order-preserving 32-bit images of the scores.
__device__ __forceinline__ uint32_t score_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_score(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
}

// Expert choice: the k largest of a row's softmax, best first, lowest position first among equals.  One CTA per row,
// a bitonic sort of 64-bit keys (score image, position).  Bound by the latency of its 66 stages at S = 2048 (the grid is
// sequences x experts, mostly less than one wave): a warp takes the strides up to 32 of 64 neighbouring keys in
// registers, so 15 stages of the 66 and one pass per size go through shared memory and a block barrier.  64 rows of 1536,
// k = 96: 23.7 -> 12.4 us.
__device__ __forceinline__ unsigned long long sort_key(float v, int i) {
  uint32_t k = score_key(v);
  if (v == 0.f) k = 0x80000000u;                     // -0 ties with +0
  if (v != v) k = 0xffffffffu;                       // NaN first, as torch.topk
  return ((unsigned long long)k << 32) | (0xffffffffu - (uint32_t)i);
}
__device__ __forceinline__ unsigned long long sort_step(unsigned long long k, int i, int size, int stride) {
  const unsigned long long o = __shfl_xor_sync(0xffffffffu, k, stride);
  const bool keep_larger = ((i & stride) == 0) == ((i & size) == 0);
  return (k > o) == keep_larger ? k : o;
}

__global__ void __launch_bounds__(1024)
seq_topk_softmax_kernel(const float* __restrict__ scores, long long row_stride, long long col_stride, int rows_inner,
                        long long outer_stride, int S, int S2, int k, long long* __restrict__ idx_out,
                        float* __restrict__ w_out, float* __restrict__ stat_out) {
  extern __shared__ unsigned long long key[];        // [S2], S2 a power of two >= 64; padding sorts last
  __shared__ float red[32];
  __shared__ float s_mx, s_den;
  const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const float* base = scores + (long long)(r / rows_inner) * outer_stride + (long long)(r % rows_inner) * row_stride;
  float mx = -CUDART_INF_F;
  for (int i = threadIdx.x; i < S2; i += blockDim.x) {
    const float v = i < S ? base[(long long)i * col_stride] : -CUDART_INF_F;
    key[i] = i < S ? sort_key(v, i) : (unsigned long long)(0xffffffffu - (uint32_t)i);
    mx = fmaxf(mx, v);
  }
  auto score = [&](int i) { return key_score((uint32_t)(key[i] >> 32)); };
  // softmax statistics of the whole row
  mx = warp_max(mx);
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    float m = lane < warps ? red[lane] : -CUDART_INF_F;
    m = warp_max(m);
    if (lane == 0) s_mx = m;
  }
  __syncthreads();
  float den = 0.f;
  for (int i = threadIdx.x; i < S; i += blockDim.x) den += __expf(score(i) - s_mx);
  den = warp_sum(den);
  if (lane == 0) red[warp] = den;
  __syncthreads();
  if (threadIdx.x < 32) {
    float d = lane < warps ? red[lane] : 0.f;
    d = warp_sum(d);
    if (lane == 0) s_den = d;
  }
  for (int size = 64; size <= S2; size <<= 1) {
    for (int stride = size >> 1; stride >= 64; stride >>= 1) {
      for (int i = threadIdx.x; i < (S2 >> 1); i += blockDim.x) {
        const int lo = 2 * i - (i & (stride - 1));
        const int hi = lo + stride;
        const unsigned long long a = key[lo], b = key[hi];
        if ((a > b) != ((lo & size) == 0)) {
          key[lo] = b;
          key[hi] = a;
        }
      }
      __syncthreads();
    }
    for (int seg = warp * 64; seg < S2; seg += warps * 64) {
      const int i0 = seg + lane, i1 = i0 + 32;
      unsigned long long k0 = key[i0], k1 = key[i1];
      if (size == 64) {
        for (int sz = 2; sz <= 32; sz <<= 1)
          for (int stride = sz >> 1; stride > 0; stride >>= 1) {
            k0 = sort_step(k0, i0, sz, stride);
            k1 = sort_step(k1, i1, sz, stride);
          }
      }
      if ((k0 > k1) != ((i0 & size) == 0)) {
        const unsigned long long t = k0;
        k0 = k1;
        k1 = t;
      }
#pragma unroll
      for (int stride = 16; stride > 0; stride >>= 1) {
        k0 = sort_step(k0, i0, size, stride);
        k1 = sort_step(k1, i1, size, stride);
      }
      key[i0] = k0;
      key[i1] = k1;
    }
    __syncthreads();
  }
  // top-k probabilities, descending; renormalised over the kept ones (+1e-9 as the reference)
  float part = 0.f;
  for (int i = threadIdx.x; i < k; i += blockDim.x) part += __expf(score(i) - s_mx) / s_den;
  part = warp_sum(part);
  if (lane == 0) red[warp] = part;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < warps; ++i) tot += red[i];
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    idx_out[(size_t)r * k + i] = (long long)(0xffffffffu - (uint32_t)key[i]);
    w_out[(size_t)r * k + i] = (__expf(score(i) - s_mx) / s_den) / (tot + 1e-9f);
  }
  if (threadIdx.x == 0) {
    stat_out[(size_t)r * 3 + 0] = s_mx;
    stat_out[(size_t)r * 3 + 1] = s_den;
    stat_out[(size_t)r * 3 + 2] = tot;
  }
}

// Mode 0 without a sort: the k-th best key of the row is found by a 4-pass radix selection over
// order-preserving 32-bit images of the scores (256-bin histograms in shared memory), then one block-wide
// prefix count places the kept positions in ascending order.  Keys compare by value
// descending and index ascending, so of the scores equal to the threshold the lowest
// positions are kept.  (The images order -0.0 below +0.0.)
__global__ void __launch_bounds__(1024)
seq_topk_select_kernel(const float* __restrict__ scores, long long row_stride, long long col_stride, int rows_inner,
                       long long outer_stride, int S, int k, long long* __restrict__ idx_out,
                       float* __restrict__ w_out) {
  extern __shared__ uint32_t ukey[];                 // [S]
  __shared__ int hist[256];
  __shared__ int warp_tot[32];
  __shared__ float red[32];
  __shared__ uint32_t s_prefix, s_top;
  __shared__ int s_need;
  const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const float* base = scores + (long long)(r / rows_inner) * outer_stride + (long long)(r % rows_inner) * row_stride;
  uint32_t mxk = 0;
  for (int i = tid; i < S; i += 1024) {
    const uint32_t u = score_key(base[(long long)i * col_stride]);
    ukey[i] = u;
    mxk = max(mxk, u);
  }
  mxk = __reduce_max_sync(0xffffffffu, mxk);
  if (lane == 0) warp_tot[wid] = (int)mxk;
  if (tid == 0) { s_prefix = 0u; s_need = k; }
  __syncthreads();
  if (wid == 0) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, (uint32_t)warp_tot[lane]);
    if (lane == 0) s_top = m;
  }
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    const uint32_t prefix = s_prefix;
    const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    for (int i = tid; i < S; i += 1024) {
      const uint32_t u = ukey[i];
      if ((u & mask) == prefix) atomicAdd(&hist[(u >> shift) & 255u], 1);
    }
    __syncthreads();
    if (wid == 0) {
      // lane L owns bins 8L .. 8L+7; the wanted key lies in the bin where the count from the top reaches `need`
      int c[8], tot = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) { c[j] = hist[8 * lane + j]; tot += c[j]; }
      int suf = tot;                                 // sum over this and all higher lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += t;
      }
      const int need = s_need;
      int above = suf - tot;
      if (above < need && need <= suf) {
#pragma unroll
        for (int j = 7; j >= 0; --j) {
          if (above < need && above + c[j] >= need) {
            s_prefix = prefix | ((uint32_t)(8 * lane + j) << shift);
            s_need = need - above;
            above = need;                            // taken: no lower bin matches
          } else {
            above += c[j];
          }
        }
      }
    }
    __syncthreads();
  }
  const uint32_t thr = s_prefix;
  const int need = s_need;                           // how many of the scores equal to the threshold are kept
  // exclusive prefix counts (greater in the low half-word, equal in the high one) over contiguous chunks
  const int per = (S + 1023) / 1024;
  const int b0 = tid * per, b1 = min(b0 + per, S);
  int packed = 0;
  for (int i = b0; i < b1; ++i) {
    const uint32_t u = ukey[i];
    packed += (u > thr ? 1 : 0) + (u == thr ? 0x10000 : 0);
  }
  int inc = packed;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_tot[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const int w = warp_tot[lane];
    int winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    warp_tot[lane] = winc - w;
  }
  __syncthreads();
  const int excl = warp_tot[wid] + inc - packed;
  int g = excl & 0xffff, e = excl >> 16;
  const float top = key_score(s_top);
  float den = 0.f;
  for (int i = b0; i < b1; ++i) {
    const uint32_t u = ukey[i];
    const bool eq = u == thr;
    if (u > thr || (eq && e < need)) {
      const int o = g + min(e, need);
      const float ex = __expf(key_score(u) - top);
      idx_out[(size_t)r * k + o] = i;
      w_out[(size_t)r * k + o] = ex;                 // normalised below
      den += ex;
    }
    g += (u > thr) ? 1 : 0;
    e += eq ? 1 : 0;
  }
  den = warp_sum(den);
  if (lane == 0) red[wid] = den;
  __threadfence_block();
  __syncthreads();
  float tot = 0.f;
#pragma unroll 8
  for (int i = 0; i < 32; ++i) tot += red[i];
  for (int i = tid; i < k; i += 1024) w_out[(size_t)r * k + i] /= tot;
}

// mode 0: dscore[idx_j] = w_j (dw_j - sum_l w_l dw_l), zero elsewhere.
// mode 1: p = softmax(row); w_j = p_j / (tot + eps); dp_j = (dw_j - sum_l dw_l w_l) / (tot + eps);
//         dscore_t = p_t (dp_t - sum_j p_j dp_j)   (dp = 0 for tokens that were not picked)
__global__ void seq_topk_bwd_kernel(const float* __restrict__ scores, long long row_stride, long long col_stride,
                                    int rows_inner, long long outer_stride, int S, int k, int mode,
                                    const long long* __restrict__ idx, const float* __restrict__ w,
                                    const float* __restrict__ dw, const float* __restrict__ stat,
                                    float* __restrict__ dscores) {
  extern __shared__ float sm[];                      // [S] dp per position (mode 1) / output staging
  __shared__ float red[32];
  const int r = blockIdx.x;
  const long long boff = (long long)(r / rows_inner) * outer_stride + (long long)(r % rows_inner) * row_stride;
  for (int i = threadIdx.x; i < S; i += blockDim.x) sm[i] = 0.f;
  float dot = 0.f;
  for (int j = threadIdx.x; j < k; j += blockDim.x) dot += w[(size_t)r * k + j] * dw[(size_t)r * k + j];
  dot = warp_sum(dot);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) tot += red[i];
  __syncthreads();
  if (mode == 0) {
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
      const float wj = w[(size_t)r * k + j];
      sm[(int)idx[(size_t)r * k + j]] = wj * (dw[(size_t)r * k + j] - tot);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < S; i += blockDim.x) dscores[boff + (long long)i * col_stride] = sm[i];
    return;
  }
  const float mx = stat[(size_t)r * 3], den = stat[(size_t)r * 3 + 1], keep = stat[(size_t)r * 3 + 2] + 1e-9f;
  float pd = 0.f;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    const int t = (int)idx[(size_t)r * k + j];
    const float dp = (dw[(size_t)r * k + j] - tot) / keep;
    sm[t] = dp;
    pd += (__expf(scores[boff + (long long)t * col_stride] - mx) / den) * dp;
  }
  pd = warp_sum(pd);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = pd;
  __syncthreads();
  float pdt = 0.f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) pdt += red[i];
  for (int i = threadIdx.x; i < S; i += blockDim.x) {
    const float p = __expf(scores[boff + (long long)i * col_stride] - mx) / den;
    dscores[boff + (long long)i * col_stride] = p * (sm[i] - pdt);
  }
}

}  // namespace kmoe

using namespace kmoe;

static int next_pow2(int x) {
  int p = 1;
  while (p < x) p <<= 1;
  return p;
}

static int route_grid(int T, int per_warp) {
  const int warps = (T + per_warp - 1) / per_warp;
  const int g = (warps + ROUTE_WARPS - 1) / ROUTE_WARPS;
  return g < 148 * 12 ? g : 148 * 12;
}

extern "C" int kmoe_route_topk_fwd(const void* logits, int is_bf16, int T, int E, int k, float* w, void* w_out,
                                   long long* idx, float* lse, float* acc, float* aux, float w_lb, float w_z,
                                   cudaStream_t st) {
  if (E > ROUTE_MAX_E || k > ROUTE_MAX_K || k > E) return -1;
  if (T == 0) return 0;
  // two tokens per warp: each CTA adds 2 E + 1 sums to the same addresses at its end
  if (is_bf16)
    route_topk_fwd_kernel<__nv_bfloat16><<<route_grid(T, 2), 32 * ROUTE_WARPS, 0, st>>>(
        (const __nv_bfloat16*)logits, T, E, k, w, (__nv_bfloat16*)w_out, idx, lse, acc, acc + E, acc + 2 * E);
  else
    route_topk_fwd_kernel<float><<<route_grid(T, 2), 32 * ROUTE_WARPS, 0, st>>>((const float*)logits, T, E, k, w,
                                                                               (float*)w_out, idx, lse, acc, acc + E,
                                                                               acc + 2 * E);
  route_aux_kernel<<<1, 32, 0, st>>>(acc, E, w_lb * (float)E / ((float)T * (float)T * (float)k), w_z / (float)T, aux);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_route_topk_bwd(const void* logits, int is_bf16, const float* lse, const long long* idx,
                                   const float* w, const void* dw, const float* counts, const float* d_aux, float w_lb,
                                   float w_z, int T, int E, int k, void* dlogits, cudaStream_t st) {
  if (E > ROUTE_MAX_E || k > ROUTE_MAX_K) return -1;
  if (T == 0) return 0;
  if (is_bf16)
    route_topk_bwd_kernel<__nv_bfloat16><<<route_grid(T, 1), 32 * ROUTE_WARPS, 0, st>>>(
        (const __nv_bfloat16*)logits, lse, idx, w, (const __nv_bfloat16*)dw, counts, d_aux, w_lb, w_z, T, E, k,
        (__nv_bfloat16*)dlogits);
  else
    route_topk_bwd_kernel<float><<<route_grid(T, 1), 32 * ROUTE_WARPS, 0, st>>>(
        (const float*)logits, lse, idx, w, (const float*)dw, counts, d_aux, w_lb, w_z, T, E, k, (float*)dlogits);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_seq_topk_fwd(const float* scores, long long row_stride, long long col_stride, int rows_inner,
                                 long long outer_stride, int rows, int S, int k, int mode, long long* idx, float* w,
                                 float* stat, cudaStream_t st) {
  const int S2 = next_pow2(S < 64 ? 64 : S);
  if (k < 1 || k > S || S2 > 16384) return -1;
  if (rows == 0) return 0;
  const size_t smem = (size_t)S2 * 8;
  static SmemLimit limit_sort, limit_select;
  if (!limit_sort.raise(seq_topk_softmax_kernel, 16384 * 8) || !limit_select.raise(seq_topk_select_kernel, 16384 * 4)) return -3;
  if (mode == 0) {      // kept positions in ascending order: selection instead of a sort
    seq_topk_select_kernel<<<rows, 1024, (size_t)S * 4, st>>>(scores, row_stride, col_stride, rows_inner,
                                                              outer_stride, S, k, idx, w);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  seq_topk_softmax_kernel<<<rows, 1024, smem, st>>>(scores, row_stride, col_stride, rows_inner, outer_stride, S, S2, k,
                                                    idx, w, stat);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_seq_topk_bwd(const float* scores, long long row_stride, long long col_stride, int rows_inner,
                                 long long outer_stride, int rows, int S, int k, int mode, const long long* idx,
                                 const float* w, const float* dw, const float* stat, float* dscores, cudaStream_t st) {
  if (S > 16384) return -1;
  if (rows == 0) return 0;
  static SmemLimit limit;
  if (!limit.raise(seq_topk_bwd_kernel, 16384 * 4)) return -3;
  seq_topk_bwd_kernel<<<rows, 512, (size_t)S * 4, st>>>(scores, row_stride, col_stride, rows_inner, outer_stride, S, k,
                                                        mode, idx, w, dw, stat, dscores);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
