// Mamba kernels, channels-last: depthwise causal conv1d (+SiLU), forward and backward (the selective
// scan lives in scan.cu).  Activations are bf16 [B, S, C] (row strides allowed where a
// tensor is a column slice of a fused projection); the small per-channel parameters
// (conv taps, bias, A, D, dt bias) and the per-step B/C vectors are fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kmoe_api.h"
#include "ptx.cuh"

namespace kmoe {

__device__ __forceinline__ float bf2f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }

// ------------------------------------------------------------------ conv1d
// y[b,t,c] = act(bias[c] + sum_j w[c,j] * x[b, t-(W-1)+j, c]),  W = 4
// A thread owns V neighbouring channels (two where rows are 4-byte aligned: a warp then moves whole 128-byte lines) and
// CONV_T steps, a CTA eight such stretches.  Both directions stream their operands once; what counts is to have enough
// loads in flight, so the rows of a batch of steps are requested, unconditionally (rows past the end repeat the last
// one), before the first of them is looked at.
// 4 x 2048 x 4096: forward 39.4 us (20.5 at the copy rate), backward 77.0 us (30.8).  What bounds both is the latency of a
// batch of loads and the arithmetic on it, one after the other: neither the issue slots (68 and 58 % busy) nor memory (DRAM
// at 29 and 27 %) is full.  The backward kernel, fourteen multiply-adds per element, took 88.0 us on single floats
// instead of packed pairs (three CTAs per SM).  The forward kernel, four per element, keeps single floats: 40.3 to 42.4 us
// on pairs (three to six CTAs).  A batch loaded ahead costs the registers of a CTA: 43 and 81 us.  Where all CTAs run at once
// the longer latency of the pairs shows: 1 x 333 x 1536 backward 11.1 us for 10.7, with its two zero fills.
constexpr int CONV_T = 32;      // time steps per thread
constexpr int CONV_WARPS = 8;

// The values P of a thread's V channels at one step: a float or a packed pair, two channels for the arithmetic
// instructions of one.
template <int V>
struct ConvVec;
template <>
struct ConvVec<1> {
  using Raw = unsigned short;
  using P = float;
  __device__ static __forceinline__ Raw load(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const Raw*>(p)); }
  __device__ static __forceinline__ P widen(Raw r) { return __uint_as_float((uint32_t)r << 16); }
  __device__ static __forceinline__ void store(__nv_bfloat16* p, P v) { *p = __float2bfloat16(v); }
  __device__ static __forceinline__ P fma(P a, P b, P c) { return fmaf(a, b, c); }
  __device__ static __forceinline__ P mul(P a, P b) { return a * b; }
  __device__ static __forceinline__ P add(P a, P b) { return a + b; }
  __device__ static __forceinline__ P zero() { return 0.f; }
  __device__ static __forceinline__ P gather(const float* p, int stride) { return p[0]; }
  template <class F>
  __device__ static __forceinline__ P map(P v, F f) { return f(v); }
  __device__ static __forceinline__ void spread(P v, float (&o)[1]) { o[0] = v; }
};
template <>
struct ConvVec<2> {
  using Raw = uint32_t;
  using P = uint64_t;
  __device__ static __forceinline__ Raw load(const __nv_bfloat16* p) { return __ldg(reinterpret_cast<const Raw*>(p)); }
  __device__ static __forceinline__ P widen(Raw r) {
    return pack_f32x2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u));
  }
  __device__ static __forceinline__ void store(__nv_bfloat16* p, P v) {
    float a, b;
    unpack_f32x2(v, a, b);
    *reinterpret_cast<uint32_t*>(p) = pack_bf16(a, b);
  }
  __device__ static __forceinline__ P fma(P a, P b, P c) { return fma_f32x2(a, b, c); }
  __device__ static __forceinline__ P mul(P a, P b) { return mul_f32x2(a, b); }
  __device__ static __forceinline__ P add(P a, P b) { return add_f32x2(a, b); }
  __device__ static __forceinline__ P zero() { return 0ull; }
  __device__ static __forceinline__ P gather(const float* p, int stride) { return pack_f32x2(p[0], p[stride]); }
  template <class F>
  __device__ static __forceinline__ P map(P v, F f) {
    float a, b;
    unpack_f32x2(v, a, b);
    return pack_f32x2(f(a), f(b));
  }
  __device__ static __forceinline__ void spread(P v, float (&o)[2]) { unpack_f32x2(v, o[0], o[1]); }
};

template <int V>
__global__ void __launch_bounds__(32 * CONV_WARPS)
conv1d_fwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                  __nv_bfloat16* __restrict__ y, int S, int C, long long ldx, int act, int bpg) {
  const int c = (blockIdx.x * 32 + (threadIdx.x & 31)) * V;
  const int t0 = (blockIdx.y * CONV_WARPS + (threadIdx.x >> 5)) * CONV_T;
  if (c >= C || t0 >= S) return;
  const int b = blockIdx.z;
  const int pc = (b / bpg) * C + c;   // parameter row: batch entries [g*bpg, (g+1)*bpg) use parameter set g
  using CV = ConvVec<V>;
  float wv[V][4], bs[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
#pragma unroll
    for (int j = 0; j < 4; ++j) wv[k][j] = w[(size_t)(pc + k) * 4 + j];
    bs[k] = bias ? bias[pc + k] : 0.f;
  }
  const __nv_bfloat16* xb = x + (size_t)b * S * ldx + c;
  __nv_bfloat16* yb = y + (size_t)b * S * C + c;
  float win[3][V];                    // x[t-3], x[t-2], x[t-1]
#pragma unroll
  for (int j = 0; j < 3; ++j) {
#pragma unroll
    for (int k = 0; k < V; ++k) win[j][k] = 0.f;
    if (t0 - 3 + j >= 0) CV::spread(CV::widen(CV::load(xb + (size_t)(t0 - 3 + j) * ldx)), win[j]);
  }
  constexpr int BATCH = 8;
#pragma unroll 1
  for (int tb = t0; tb < min(t0 + CONV_T, S); tb += BATCH) {
    typename CV::Raw raw[BATCH];
#pragma unroll
    for (int i = 0; i < BATCH; ++i) raw[i] = CV::load(xb + (size_t)min(tb + i, S - 1) * ldx);
    float xv[BATCH][V];
#pragma unroll
    for (int i = 0; i < BATCH; ++i) CV::spread(CV::widen(raw[i]), xv[i]);
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      float o[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const float x0 = i > 2 ? xv[i - 3][k] : win[i][k], x1 = i > 1 ? xv[i - 2][k] : win[i + 1][k],
                    x2 = i > 0 ? xv[i - 1][k] : win[2][k];
        const float v = bs[k] + wv[k][0] * x0 + wv[k][1] * x1 + wv[k][2] * x2 + wv[k][3] * xv[i][k];
        o[k] = act ? silu_f(v) : v;
      }
      if (tb + i < S) CV::store(yb + (size_t)(tb + i) * C, CV::gather(o, 1));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < V; ++k) win[j][k] = xv[BATCH - 3 + j][k];
  }
}

// dx (rows lddx apart), and atomically accumulated dw [C,4], dbias [C] (fp32, zeroed by the caller; one addition per
// channel and CTA).
template <int V>
__global__ void __launch_bounds__(32 * CONV_WARPS, 3)
conv1d_bwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                  const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, float* __restrict__ dw,
                  float* __restrict__ dbias, int S, int C, long long ldx, long long lddx, int act, int bpg) {
  __shared__ float sums[CONV_WARPS][5 * V][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * V;
  const int t0 = (blockIdx.y * CONV_WARPS + warp) * CONV_T;
  const int b = blockIdx.z;
  const int pc = (b / bpg) * C + c;
  using CV = ConvVec<V>;
  using P = typename CV::P;
  P acc[5];                           // dw[0..3], dbias
#pragma unroll
  for (int j = 0; j < 5; ++j) acc[j] = CV::zero();
  if (c < C && t0 < S) {
    P wv[4], bs = bias ? CV::gather(bias + pc, 1) : CV::zero();
#pragma unroll
    for (int j = 0; j < 4; ++j) wv[j] = CV::gather(w + (size_t)pc * 4 + j, 4);
    const __nv_bfloat16* xb = x + (size_t)b * S * ldx + c;
    const __nv_bfloat16* gb = dy + (size_t)b * S * C + c;
    __nv_bfloat16* dxb = dx + (size_t)b * S * lddx + c;
    const int t_own = min(t0 + CONV_T, S);
    P xw[3], pw[3];                   // x[t-3 .. t-1], dpre[t-3 .. t-1]; the dpre window starts empty, which is exact:
#pragma unroll                        // dx[td >= t0] never reads dpre[< t0]
    for (int j = 0; j < 3; ++j) {
      xw[j] = t0 - 3 + j >= 0 ? CV::widen(CV::load(xb + (size_t)(t0 - 3 + j) * ldx)) : CV::zero();
      pw[j] = CV::zero();
    }
    constexpr int BATCH = 7;          // CONV_T + 3 steps in all: dx[t] needs dpre up to t + 3
    static_assert((CONV_T + 3) % BATCH == 0, "whole batches");
#pragma unroll 1
    for (int tb = t0; tb < t0 + CONV_T + 3; tb += BATCH) {
      typename CV::Raw xr[BATCH], gr[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        const int t = min(tb + i, S - 1);
        xr[i] = CV::load(xb + (size_t)t * ldx);
        gr[i] = CV::load(gb + (size_t)t * C);
      }
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        const P x3 = CV::widen(xr[i]);
        P g = tb + i < S ? CV::widen(gr[i]) : CV::zero();
        if (act) {
          const P pre = CV::fma(wv[3], x3, CV::fma(wv[2], xw[2], CV::fma(wv[1], xw[1], CV::fma(wv[0], xw[0], bs))));
          g = CV::mul(g, CV::map(pre, [](float u) {
                        const float sg = sigmoid_f(u);
                        return sg * (1.f + u * (1.f - sg));
                      }));
        }
        if (tb + i < t_own) {
          acc[0] = CV::fma(g, xw[0], acc[0]);
          acc[1] = CV::fma(g, xw[1], acc[1]);
          acc[2] = CV::fma(g, xw[2], acc[2]);
          acc[3] = CV::fma(g, x3, acc[3]);
          acc[4] = CV::add(g, acc[4]);
        }
        // dx[t - 3] = w0 dpre[t] + w1 dpre[t-1] + w2 dpre[t-2] + w3 dpre[t-3]
        const P o = CV::fma(wv[0], g, CV::fma(wv[1], pw[2], CV::fma(wv[2], pw[1], CV::mul(wv[3], pw[0]))));
        xw[0] = xw[1]; xw[1] = xw[2]; xw[2] = x3;
        pw[0] = pw[1]; pw[1] = pw[2]; pw[2] = g;
        const int td = tb + i - 3;
        if (td >= t0 && td < t_own) CV::store(dxb + (size_t)td * lddx, o);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    float v[V];
    CV::spread(acc[j], v);
#pragma unroll
    for (int k = 0; k < V; ++k) sums[warp][k * 5 + j][lane] = v[k];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 5 * V * 32; i += 32 * CONV_WARPS) {
    const int kj = i / 32, l = i % 32, k = kj / 5, j = kj % 5, cc = (blockIdx.x * 32 + l) * V + k;
    if (cc >= C) continue;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < CONV_WARPS; ++q) v += sums[q][kj][l];
    const size_t row = (size_t)(b / bpg) * C + cc;
    if (j < 4) atomicAdd(&dw[row * 4 + j], v);
    else if (dbias) atomicAdd(&dbias[row], v);
  }
}

// ------------------------------------------------------------------ parameters
// The mixer's small parameters as the kernels read them, in one launch instead of a cast per tensor: flat fp32
//   A = -exp(A_log) [C,16] | conv weight [C,4] | conv bias [C] | dt bias [C] | D [C]
// Their gradients accumulate in a buffer of the same layout; the second kernel turns it into the parameters' type, with
// dA_log = dA * A.
template <typename T>
__global__ void mamba_params_kernel(const T* __restrict__ A_log, const T* __restrict__ conv_w, const T* __restrict__ conv_b,
                                    const T* __restrict__ dt_b, const T* __restrict__ D, float* __restrict__ out, int C) {
  const int n = C * 23;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float v;
    if (i < 16 * C) v = (float)-exp((double)(float)A_log[i]);   // not the fast-math expf
    else if (i < 20 * C) v = (float)conv_w[i - 16 * C];
    else if (i < 21 * C) v = (float)conv_b[i - 20 * C];
    else if (i < 22 * C) v = (float)dt_b[i - 21 * C];
    else v = (float)D[i - 22 * C];
    out[i] = v;
  }
}
template <typename T>
__global__ void mamba_params_bwd_kernel(const float* __restrict__ acc, const float* __restrict__ params,
                                        T* __restrict__ out, int C) {
  const int n = C * 23;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = (T)(i < 16 * C ? acc[i] * params[i] : acc[i]);
}
// fp32 rows dB | dC (two [rows, 16] arrays) -> the last 32 columns of bf16 rows `ld` apart
__global__ void mamba_pack_bc_kernel(const float* __restrict__ dB, const float* __restrict__ dC,
                                     __nv_bfloat16* __restrict__ out, long long rows, long long ld) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < rows * 8; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i >> 3;
    const int q = (int)(i & 7);
    const float4 v = *reinterpret_cast<const float4*>((q < 4 ? dB : dC) + r * 16 + (q & 3) * 4);
    *reinterpret_cast<uint2*>(out + r * ld + q * 4) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  }
}

static bool conv_pairs(const void* a, const void* b, const void* c, int C, long long ld1, long long ld2) {
  return C % 2 == 0 && ld1 % 2 == 0 && ld2 % 2 == 0 &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 3) == 0;
}
static dim3 conv_grid(int B, int S, int C, int v) {
  return dim3((C + 32 * v - 1) / (32 * v), (S + CONV_T * CONV_WARPS - 1) / (CONV_T * CONV_WARPS), B);
}

}  // namespace kmoe

using namespace kmoe;

extern "C" int kmoe_conv1d_fwd(const void* x, const float* w, const float* bias, void* y, int B, int S, int C,
                               long long ldx, int act, int groups, cudaStream_t st) {
  if (groups < 1 || B % groups) return -1;
  if (B == 0 || S == 0 || C == 0) return 0;
  const bool two = conv_pairs(x, y, y, C, ldx, C);
  auto kern = two ? conv1d_fwd_kernel<2> : conv1d_fwd_kernel<1>;
  kern<<<conv_grid(B, S, C, two ? 2 : 1), 32 * CONV_WARPS, 0, st>>>((const __nv_bfloat16*)x, w, bias, (__nv_bfloat16*)y, S,
                                                                    C, ldx, act, B / groups);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_conv1d_bwd(const void* x, const float* w, const float* bias, const void* dy, void* dx, float* dw,
                               float* dbias, int B, int S, int C, long long ldx, long long lddx, int act, int groups,
                               cudaStream_t st) {
  if (groups < 1 || B % groups) return -1;
  if (B == 0 || S == 0 || C == 0) return 0;
  const bool two = conv_pairs(x, dy, dx, C, ldx, lddx);
  auto kern = two ? conv1d_bwd_kernel<2> : conv1d_bwd_kernel<1>;
  kern<<<conv_grid(B, S, C, two ? 2 : 1), 32 * CONV_WARPS, 0, st>>>((const __nv_bfloat16*)x, w, bias,
                                                                    (const __nv_bfloat16*)dy, (__nv_bfloat16*)dx, dw, dbias,
                                                                    S, C, ldx, lddx, act, B / groups);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_mamba_params(const void* A_log, const void* conv_w, const void* conv_b, const void* dt_b, const void* D,
                                 int is_bf16, float* out, int C, cudaStream_t st) {
  const int grid = (C * 23 + 255) / 256;
  if (is_bf16)
    mamba_params_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)A_log, (const __nv_bfloat16*)conv_w,
                                                             (const __nv_bfloat16*)conv_b, (const __nv_bfloat16*)dt_b,
                                                             (const __nv_bfloat16*)D, out, C);
  else
    mamba_params_kernel<float><<<grid, 256, 0, st>>>((const float*)A_log, (const float*)conv_w, (const float*)conv_b,
                                                     (const float*)dt_b, (const float*)D, out, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_mamba_params_bwd(const float* acc, const float* params, void* out, int is_bf16, int C, cudaStream_t st) {
  const int grid = (C * 23 + 255) / 256;
  if (is_bf16)
    mamba_params_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(acc, params, (__nv_bfloat16*)out, C);
  else
    mamba_params_bwd_kernel<float><<<grid, 256, 0, st>>>(acc, params, (float*)out, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_mamba_pack_bc(const float* dB, const float* dC, void* out, long long rows, long long ld,
                                  cudaStream_t st) {
  if (ld % 4 || (reinterpret_cast<uintptr_t>(out) & 7)) return -1;
  if (rows <= 0) return 0;
  const long long grid = (rows * 8 + 255) / 256;
  mamba_pack_bc_kernel<<<(unsigned)(grid < 148 * 8 ? grid : 148 * 8), 256, 0, st>>>(dB, dC, (__nv_bfloat16*)out, rows, ld);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
