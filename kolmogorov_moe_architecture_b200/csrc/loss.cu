// Cross-entropy over a bf16 logits tile with the gradient written in place.
//
// The LM-head + MTP loss is evaluated head by head and row-chunk by row-chunk:
// logits = H W^T (tcgen05 GEMM), then this kernel turns the chunk into
// d(loss)/d(logits) in place while producing the per-row losses, then two more
// GEMMs consume the gradient chunk.  The chunk is the only (rows, V) tensor that
// ever exists.  One CTA per row, fp32 max / sum-exp; a row that fits in shared memory
// is read once (ce_fwd_bwd_row_kernel), a longer one twice, the second time from L2.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kmoe_api.h"
#include "ptx.cuh"

namespace kmoe {

constexpr int CE_THREADS = 256;

__device__ __forceinline__ void merge_ms(float& m, float& s, float m2, float s2) {
  if (m2 == -INFINITY) return;
  if (m == -INFINITY) {
    m = m2;
    s = s2;
    return;
  }
  const float mn = fmaxf(m, m2);
  s = s * __expf(m - mn) + s2 * __expf(m2 - mn);
  m = mn;
}

// log S + M - x in 64 bits: one value per row, and the 32-bit fast logarithm left a bias of -3.2e-7 in the rows' mean
// (2048 rows of 50257, now -6e-8; largest error 1.2e-6, now 6.4e-7) at the same time.
__device__ __forceinline__ float row_loss(float S, double M, float x) { return (float)(log((double)S) + M - (double)x); }

// logits [R, V] (ld), labels [R] int64 (already shifted / masked; ignore_index rows give zero loss and gradient)
// loss_rows [R] fp32 ; if write_grad: logits <- (softmax - onehot) * (*grad_scale)
__global__ void __launch_bounds__(CE_THREADS)
ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                  float* __restrict__ loss_rows, const float* __restrict__ grad_scale, int V, long long ld,
                  long long ignore_index, int write_grad) {
  __shared__ float sm[CE_THREADS / 32], ss[CE_THREADS / 32];
  __shared__ float s_max, s_sum;
  const int row = blockIdx.x;
  __nv_bfloat16* lr = logits + (size_t)row * ld;
  const long long label = labels[row];
  const bool ignored = (label == ignore_index) || label < 0 || label >= V;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int vec = V / 8;
  if (ignored) {
    if (tid == 0) loss_rows[row] = 0.f;
    if (write_grad) {
      for (int v = tid; v < vec; v += CE_THREADS) reinterpret_cast<uint4*>(lr)[v] = make_uint4(0, 0, 0, 0);
      for (int c = vec * 8 + tid; c < V; c += CE_THREADS) lr[c] = __float2bfloat16(0.f);
    }
    return;
  }
  float m = -INFINITY, s = 0.f;
  for (int v = tid; v < vec; v += CE_THREADS) {
    uint4 r = reinterpret_cast<const uint4*>(lr)[v];
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&r);
    float x[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(p[i]);
      x[2 * i] = f.x;
      x[2 * i + 1] = f.y;
    }
    float mx = x[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) mx = fmaxf(mx, x[i]);
    const float mn = fmaxf(m, mx);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = __expf(x[i] - mn);
    s = s * __expf(m - mn) + (((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7])));
    m = mn;
  }
  for (int c = vec * 8 + tid; c < V; c += CE_THREADS) merge_ms(m, s, __bfloat162float(lr[c]), 1.f);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    merge_ms(m, s, m2, s2);
  }
  if (lane == 0) { sm[wid] = m; ss[wid] = s; }
  __syncthreads();
  if (tid == 0) {
    float M = sm[0], S = ss[0];
    for (int w = 1; w < CE_THREADS / 32; ++w) merge_ms(M, S, sm[w], ss[w]);
    s_max = M;
    s_sum = S;
    loss_rows[row] = row_loss(S, M, __bfloat162float(lr[label]));
  }
  __syncthreads();
  if (!write_grad) return;
  const float M = s_max, inv = 1.f / s_sum, gs = *grad_scale;
  for (int v = tid; v < vec; v += CE_THREADS) {
    uint4 r = reinterpret_cast<const uint4*>(lr)[v];
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&r);
    const int c0 = v * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(p[i]);
      float g0 = __expf(f.x - M) * inv, g1 = __expf(f.y - M) * inv;
      if (c0 + 2 * i == label) g0 -= 1.f;
      if (c0 + 2 * i + 1 == label) g1 -= 1.f;
      p[i] = __floats2bfloat162_rn(g0 * gs, g1 * gs);
    }
    reinterpret_cast<uint4*>(lr)[v] = r;
  }
  for (int c = vec * 8 + tid; c < V; c += CE_THREADS) {
    float g = __expf(__bfloat162float(lr[c]) - M) * inv;
    if (c == label) g -= 1.f;
    lr[c] = __float2bfloat16(g * gs);
  }
}

// The same with the row kept in shared memory: one read and one write of the logits.  In the kernel above the second pass
// is meant to hit L2, but the rows of all resident CTAs (about 1200 x 100 KB at V = 50257) are as large as the L2, and it
// mostly does not.  Two 512-thread CTAs per SM up to V = 56 k, one up to V = 114 k.  4096 x 50257: 214 -> 186 us per
// head; 126 us at the copy rate, about 100 us for the two exponentials per element.
constexpr int CE_ROW_THREADS = 512;
constexpr int CE_ROW_MAX = 225 * 1024;      // bytes of a row

__device__ __forceinline__ float ce_block_reduce(float v, float* sm, bool is_max) {
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();                           // the previous reduction's result has been read
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = sm[0];
#pragma unroll
  for (int w = 1; w < CE_ROW_THREADS / 32; ++w) r = is_max ? fmaxf(r, sm[w]) : r + sm[w];
  return r;
}

__global__ void __launch_bounds__(CE_ROW_THREADS, 2)
ce_fwd_bwd_row_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                      float* __restrict__ loss_rows, const float* __restrict__ grad_scale, int V, long long ld,
                      long long ignore_index, int write_grad) {
  extern __shared__ __align__(16) uint8_t ce_row[];
  __shared__ float red[CE_ROW_THREADS / 32];
  uint4* sr = reinterpret_cast<uint4*>(ce_row);
  __nv_bfloat16* srow = reinterpret_cast<__nv_bfloat16*>(ce_row);
  const int row = blockIdx.x, tid = threadIdx.x;
  __nv_bfloat16* lr = logits + (size_t)row * ld;
  const long long label = labels[row];
  const bool ignored = (label == ignore_index) || label < 0 || label >= V;
  const int vec = V / 8;
  if (ignored) {
    if (tid == 0) loss_rows[row] = 0.f;
    if (write_grad) {
      for (int v = tid; v < vec; v += CE_ROW_THREADS) reinterpret_cast<uint4*>(lr)[v] = make_uint4(0, 0, 0, 0);
      for (int c = vec * 8 + tid; c < V; c += CE_ROW_THREADS) lr[c] = __float2bfloat16(0.f);
    }
    return;
  }
  auto widen = [](const uint4& r, float (&x)[8]) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[2 * i] = __uint_as_float(w[i] << 16);
      x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  };
  float m = -INFINITY;
#pragma unroll 4
  for (int v = tid; v < vec; v += CE_ROW_THREADS) {
    const uint4 r = __ldcs(reinterpret_cast<const uint4*>(lr) + v);
    sr[v] = r;
    float x[8];
    widen(r, x);
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, x[i]);
  }
  for (int c = vec * 8 + tid; c < V; c += CE_ROW_THREADS) {
    srow[c] = lr[c];
    m = fmaxf(m, __bfloat162float(srow[c]));
  }
  const float M = ce_block_reduce(m, red, true);
  // e^(x - M) = 2^(x log2(e) - M log2(e)) as one fused multiply-add and one MUFU instruction; what rounding M log2(e)
  // costs is a factor common to all entries and drops out of the quotient
  constexpr float L2E = 1.4426950408889634f;
  const float nM = -M * L2E;
  float s = 0.f;
#pragma unroll 2
  for (int v = tid; v < vec; v += CE_ROW_THREADS) {
    float x[8];
    widen(sr[v], x);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = ex2_approx(fmaf(x[i], L2E, nM));
    s += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
  }
  for (int c = vec * 8 + tid; c < V; c += CE_ROW_THREADS) s += ex2_approx(fmaf(__bfloat162float(srow[c]), L2E, nM));
  const float S = ce_block_reduce(s, red, false);
  // the M of the exponentials, nM / -log2(e)
  if (tid == 0) loss_rows[row] = row_loss(S, (double)nM * -0.6931471805599453, __bfloat162float(srow[label]));
  if (!write_grad) return;
  const float gs = *grad_scale, f = gs / S;
#pragma unroll 2
  for (int v = tid; v < vec; v += CE_ROW_THREADS) {
    float x[8];
    widen(sr[v], x);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = ex2_approx(fmaf(x[i], L2E, nM)) * f;
    if ((int)label >> 3 == v) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (((int)label & 7) == i) x[i] -= gs;
    }
    reinterpret_cast<uint4*>(lr)[v] =
        make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
  }
  for (int c = vec * 8 + tid; c < V; c += CE_ROW_THREADS) {
    const float g = ex2_approx(fmaf(__bfloat162float(srow[c]), L2E, nM)) * f;
    lr[c] = __float2bfloat16(c == label ? g - gs : g);
  }
}

// The multi-token loss around the rows, one small kernel on either side of them (as single tensor operations they were
// 45 launches and 165 us of 6.7 ms for four heads of 4096 tokens, now 13 us).
// Head h = blockIdx.x: the label of each token for it (h + 1 places on in its sequence of S, none: ignore_index), how many
// it has to predict, and what a row's gradient is scaled by.  The rows' kernel reads its label from the table: found in
// the row itself (a remainder per thread) it took 193 us instead of 182 for 4096 rows of 50257.
__global__ void __launch_bounds__(1024) mtp_labels_kernel(const long long* __restrict__ labels, int R, int S,
                                                          long long ignore_index, const float* __restrict__ weights,
                                                          long long* __restrict__ shifted, float* __restrict__ n_valid,
                                                          float* __restrict__ grad_scale) {
  __shared__ int red[32];
  const int shift = blockIdx.x + 1;
  int n = 0;
  for (int t = threadIdx.x; t < R; t += 1024) {
    const long long l = t % S + shift < S ? labels[t + shift] : ignore_index;
    shifted[(size_t)blockIdx.x * R + t] = l;
    n += l != ignore_index ? 1 : 0;
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x < 32) {
    n = __reduce_add_sync(0xffffffffu, red[threadIdx.x]);
    if (threadIdx.x == 0) {
      const float v = (float)(n < 1 ? 1 : n);
      n_valid[blockIdx.x] = v;
      grad_scale[blockIdx.x] = __fdiv_rn(weights[blockIdx.x], v);
    }
  }
}

// per[h] = sum of head h's R row losses / n_valid[h] (0 for a head that no token has a label for: h >= scored),
// total = sum of weights[h] * per[h].  Sums in 64 bits, in a fixed order.
__global__ void __launch_bounds__(1024) mtp_total_kernel(const float* __restrict__ loss_rows, long long R, int heads,
                                                         int scored, const float* __restrict__ weights,
                                                         const float* __restrict__ n_valid, float* __restrict__ per,
                                                         float* __restrict__ total) {
  __shared__ double red[32];
  float sum = 0.f;
  for (int h = 0; h < heads; ++h) {
    double s = 0;
    if (h < scored)
      for (long long r = threadIdx.x; r < R; r += 1024) s += (double)loss_rows[h * R + r];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      s = 0;
      for (int w = 0; w < 32; ++w) s += red[w];
      const float v = h < scored ? (float)(s / n_valid[h]) : 0.f;
      per[h] = v;
      sum += weights[h] * v;
    }
  }
  if (threadIdx.x == 0) *total = sum;
}

}  // namespace kmoe

extern "C" int kmoe_mtp_labels(const long long* labels, long long R, int S, int heads, long long ignore_index,
                               const float* weights, long long* shifted, float* n_valid, float* grad_scale,
                               cudaStream_t st) {
  if (R < 0 || R >= (1LL << 31) - 1024 || heads <= 0) return -1;
  kmoe::mtp_labels_kernel<<<heads, 1024, 0, st>>>(labels, (int)R, S, ignore_index, weights, shifted, n_valid, grad_scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_mtp_total(const float* loss_rows, long long R, int heads, int scored, const float* weights,
                              const float* n_valid, float* per, float* total, cudaStream_t st) {
  kmoe::mtp_total_kernel<<<1, 1024, 0, st>>>(loss_rows, R, heads, scored, weights, n_valid, per, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_ce_fwd_bwd(void* logits, const long long* labels, float* loss_rows, const float* grad_scale,
                               int R, int V, long long ld, long long ignore_index, int write_grad, cudaStream_t st) {
  if (ld % 8) return -1;
  if (R <= 0) return 0;
  const int row_bytes = (V * 2 + 15) / 16 * 16;
  if (row_bytes <= kmoe::CE_ROW_MAX && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
    static kmoe::SmemLimit limit;
    if (!limit.raise(kmoe::ce_fwd_bwd_row_kernel, kmoe::CE_ROW_MAX)) return -3;
    kmoe::ce_fwd_bwd_row_kernel<<<R, kmoe::CE_ROW_THREADS, row_bytes, st>>>((__nv_bfloat16*)logits, labels, loss_rows,
                                                                            grad_scale, V, ld, ignore_index, write_grad);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
  }
  kmoe::ce_fwd_bwd_kernel<<<R, kmoe::CE_THREADS, 0, st>>>((__nv_bfloat16*)logits, labels, loss_rows, grad_scale, V, ld,
                                                          ignore_index, write_grad);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
