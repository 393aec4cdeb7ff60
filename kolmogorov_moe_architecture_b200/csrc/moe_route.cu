// Token-choice MoE bookkeeping without host synchronisation.
//
// Layout ("padded expert-major"): the assignments of expert e occupy rows
// [off[e], off[e] + cnt[e]) of a [max_rows, d] buffer, with off[e] a multiple of 128,
// so a 128-row GEMM tile never spans two experts; rows between cnt[e] and the next
// multiple of 128 are zero.  Within an expert, rows keep (token, slot) order - the
// sort is stable, so results are deterministic.  max_rows = T*k + E*127 rounded up
// is a static bound, which keeps every buffer shape fixed across steps.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kmoe_api.h"
#include "ptx.cuh"

namespace kmoe {

constexpr int PLAN_THREADS = 256;
constexpr int ROW_TILE = 128;

// Single-block stable counting sort of n = T*k assignments over E experts.
//   idx      [n] int64 expert of each assignment (flat (token, slot) order)
//   keep     [n] bool/uint8 or null: 0 = dropped assignment
//   pos      [n] int32  row of the assignment in the padded layout, -1 if dropped
//   row_src  [max_rows] int32 flat assignment index feeding each row, -1 for padding
//   counts   [E] int32 ; offsets [E+1] int32 (padded) ; tile_group [max_rows/128] ; meta[0] = live m-tiles,
//   meta[1] = live padded rows
//
// 32 warps with a contiguous stretch of assignments each.  A warp takes 32 assignments at a time: lanes with the same
// expert find each other with match_any, their rank is the lane order, and the first of them advances the warp's count of
// that expert.  First pass: counts; then an exclusive scan over the warps per expert; second pass: rows.  256 threads that
// walked a private stretch each, with a histogram per thread, took 29 us for 12288 assignments of 16 experts (33 for 64
// experts); this way 17 us (14).
constexpr int PLAN_WARPS = 32;
__global__ void __launch_bounds__(32 * PLAN_WARPS)
moe_plan_kernel(const long long* __restrict__ idx, const unsigned char* __restrict__ keep, int n, int E, int max_rows,
                int expert_base, int* __restrict__ pos, int* __restrict__ row_src, int* __restrict__ counts,
                int* __restrict__ offsets, int* __restrict__ tile_group, int* __restrict__ meta) {
  extern __shared__ int sh[];                 // run[PLAN_WARPS][E], off[E + 1]
  int* off = sh + PLAN_WARPS * E;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* run = sh + warp * E;                   // this warp's next rank of every expert
  const int seg = (n + 32 * PLAN_WARPS - 1) / (32 * PLAN_WARPS) * 32;
  const int lo = min(warp * seg, n), hi = min(lo + seg, n);
  auto local_expert = [&](int i) -> int {     // E: not routed to an expert of this plan
    if (i >= hi) return E;
    const long long e = idx[i] - expert_base;
    return (e >= 0 && e < E && (keep == nullptr || keep[i])) ? (int)e : E;
  };
  for (int i = tid; i < PLAN_WARPS * E; i += 32 * PLAN_WARPS) sh[i] = 0;
  for (int i = tid; i < max_rows; i += 32 * PLAN_WARPS) row_src[i] = -1;
  __syncthreads();
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int e = local_expert(i0 + lane);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e < E && (same & ((1u << lane) - 1)) == 0) run[e] += __popc(same);
    __syncwarp();
  }
  __syncthreads();
  for (int e = tid; e < E; e += 32 * PLAN_WARPS) {
    int sum = 0;
    for (int w = 0; w < PLAN_WARPS; ++w) {
      const int v = sh[w * E + e];
      sh[w * E + e] = sum;
      sum += v;
    }
    counts[e] = sum;
    off[e] = sum;                             // temporarily the count
  }
  __syncthreads();
  if (warp == 0) {
    // exclusive scan of the padded counts, 32 experts at a time
    int base = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int rows = e < E ? (off[e] + ROW_TILE - 1) / ROW_TILE * ROW_TILE : 0;
      int inc = rows;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (e < E) {
        off[e] = base + inc - rows;
        offsets[e] = base + inc - rows;
        for (int j = 0; j < rows / ROW_TILE; ++j) tile_group[(base + inc - rows) / ROW_TILE + j] = e;
      }
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
    for (int j = base / ROW_TILE + lane; j < max_rows / ROW_TILE; j += 32) tile_group[j] = 0;
    if (lane == 0) {
      offsets[E] = base;
      meta[0] = base / ROW_TILE;
      meta[1] = base;
    }
  }
  __syncthreads();
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane, e = local_expert(i);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    int p = -1;
    if (e < E) {
      p = off[e] + run[e] + __popc(same & ((1u << lane) - 1));
      if (p < max_rows) row_src[p] = i; else p = -1;
    }
    __syncwarp();
    if (e < E && (same & ((1u << lane) - 1)) == 0) run[e] += __popc(same);
    __syncwarp();
    if (i < hi) pos[i] = p;
  }
}

// Capacity with drops for token choice: keep[i] = 1 iff assignment i is among the first `cap` assignments of its
// expert in flat (token, slot) order.  Same single-block stable ranking as the plan kernel.
__global__ void __launch_bounds__(PLAN_THREADS)
moe_capacity_mask_kernel(const long long* __restrict__ idx, int n, int E, int cap, unsigned char* __restrict__ keep) {
  extern __shared__ int sh[];     // hist[PLAN_THREADS][E]
  int* hist = sh;
  const int tid = threadIdx.x;
  const int seg = (n + PLAN_THREADS - 1) / PLAN_THREADS;
  const int lo = min(tid * seg, n), hi = min(lo + seg, n);
  for (int e = 0; e < E; ++e) hist[tid * E + e] = 0;
  for (int i = lo; i < hi; ++i) {
    const int e = (int)idx[i];
    if (e >= 0 && e < E) hist[tid * E + e]++;
  }
  __syncthreads();
  for (int e = tid; e < E; e += PLAN_THREADS) {
    int run = 0;
    for (int t = 0; t < PLAN_THREADS; ++t) {
      const int v = hist[t * E + e];
      hist[t * E + e] = run;
      run += v;
    }
  }
  __syncthreads();
  for (int i = lo; i < hi; ++i) {
    const int e = (int)idx[i];
    keep[i] = (e >= 0 && e < E && hist[tid * E + e]++ < cap) ? 1 : 0;
  }
}

// One slot of the balanced token-choice assignment: every token takes its most probable expert among those it
// has not used and that were not full (count >= cap) when the slot began; a token whose unused experts are all
// full takes its most probable unused expert regardless.  One warp per token; ties go to the lower index.
//   taken [T, E] uint8 (in/out), counts_in [E] (read), counts_out [E] (incremented), sel [T] int64
__global__ void moe_balanced_slot_kernel(const float* __restrict__ probs, unsigned char* __restrict__ taken,
                                         const int* __restrict__ counts_in, int* __restrict__ counts_out,
                                         long long* __restrict__ sel, long long sel_stride, int T, int E, int cap) {
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < T; t += warps) {
    float best = -INFINITY, fb = -INFINITY;
    int bi = E, fi = E;
    for (int e = lane; e < E; e += 32) {
      if (taken[(size_t)t * E + e]) continue;
      const float p = probs[(size_t)t * E + e];
      if (p > fb) { fb = p; fi = e; }
      if (counts_in[e] < cap && p > best) { best = p; bi = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o), of = __shfl_xor_sync(0xffffffffu, fb, o);
      const int obi = __shfl_xor_sync(0xffffffffu, bi, o), ofi = __shfl_xor_sync(0xffffffffu, fi, o);
      if (ob > best || (ob == best && obi < bi)) { best = ob; bi = obi; }
      if (of > fb || (of == fb && ofi < fi)) { fb = of; fi = ofi; }
    }
    const int pick = bi < E ? bi : (fi < E ? fi : 0);
    if (lane == 0) {
      sel[(size_t)t * sel_stride] = pick;
      taken[(size_t)t * E + pick] = 1;
      atomicAdd(&counts_out[pick], 1);
    }
  }
}

// dst[row] = src[row_src[row] / div]  (zero for padding rows), rows < meta[1].
__global__ void moe_gather_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ row_src,
                                       const int* __restrict__ meta, __nv_bfloat16* __restrict__ dst, int max_rows,
                                       int d, int div) {
  const int live_rows = min(meta[1], max_rows);
  const int vec = d / 8;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < live_rows; row += warps) {
    const int a = row_src[row];
    uint4* drow = reinterpret_cast<uint4*>(dst + (size_t)row * d);
    if (a < 0) {
      for (int v = lane; v < vec; v += 32) drow[v] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* srow = reinterpret_cast<const uint4*>(src + (size_t)(a / div) * d);
    for (int v = lane; v < vec; v += 32) drow[v] = srow[v];
  }
}

// out[t] = sum_k w[t,k] * Y[pos[t,k]]   (pos < 0 skipped; w null = 1).  Bound by memory latency: one warp per 512 columns
// of a token, two rows of it in flight (a lane holds four 16-byte loads), added in slot order.  Expert choice calls this
// with k = experts and mostly empty slots, a few tokens having many; a whole row per warp made those the tail of the
// launch.  6144 x 2048: two rows each 16.4 -> 15.1 us (26 with one load per lane), one row each among 16 slots 20.7 ->
// 13.5 us.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16* __restrict__ Y, const int* __restrict__ pos, const float* __restrict__ w,
                   __nv_bfloat16* __restrict__ out, int T, int k, int d) {
  constexpr int U = 2;
  const int vec = d / 8;
  const int chunks = (vec + 32 * U - 1) / (32 * U);
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (long long wi = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; wi < (long long)T * chunks; wi += warps) {
    const int t = (int)(wi / chunks);
    const int v0 = (int)(wi - (long long)t * chunks) * 32 * U + lane;
    float acc[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[u][i] = 0.f;
    for (int j0 = 0; j0 < k; j0 += 32) {
      const int pj = j0 + lane < k ? pos[(size_t)t * k + j0 + lane] : -1;
      const float wj = (w != nullptr && pj >= 0) ? w[(size_t)t * k + j0 + lane] : 1.f;
      unsigned m = __ballot_sync(0xffffffffu, pj >= 0);
      while (m != 0) {
        int p[2];
        float s[2];
        uint4 r[2][U];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int j = m != 0 ? __ffs(m) - 1 : -1;
          m &= m - 1;
          p[q] = __shfl_sync(0xffffffffu, pj, j & 31);
          s[q] = __shfl_sync(0xffffffffu, wj, j & 31);
          if (j < 0) p[q] = -1;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32;
            r[q][u] = p[q] >= 0 && v < vec ? __ldg(reinterpret_cast<const uint4*>(Y + (size_t)p[q] * d) + v)
                                           : make_uint4(0, 0, 0, 0);
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (p[q] < 0) break;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&r[q][u]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = __bfloat1622float2(b[i]);
              acc[u][2 * i] += s[q] * f.x;
              acc[u][2 * i + 1] += s[q] * f.y;
            }
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = v0 + u * 32;
      if (v < vec)
        *reinterpret_cast<uint4*>(out + (size_t)t * d + v * 8) =
            make_uint4(pack_bf16(acc[u][0], acc[u][1]), pack_bf16(acc[u][2], acc[u][3]), pack_bf16(acc[u][4], acc[u][5]),
                       pack_bf16(acc[u][6], acc[u][7]));
    }
  }
}

// Backward of the weighted combine in one pass over the rows: dY[row] = w[a] * dout[t] and dw = <dout[t], Y[row]>, with
// a = row_src[row] and t = a / k.  Bound by memory; as two kernels dout's rows were read twice and the dot products ran
// over k slots per token although only the rows exist.  One warp per row, four loads of each side in flight.
// dw is written at a (assignments without a row: 0), or, where C > 0 (expert choice: B sequences, C picks each, rows in
// (expert, sequence, pick) order), at (sequence, expert, pick).
// Against the two kernels: 12288 rows of 2048 33.5 -> 22.5 us, 6144 rows among 16 slots 35 -> 14.8 us.
__global__ void __launch_bounds__(256)
moe_gather_dw_kernel(const __nv_bfloat16* __restrict__ dout, const int* __restrict__ row_src, const float* __restrict__ w,
                     const __nv_bfloat16* __restrict__ Y, const int* __restrict__ meta, const int* __restrict__ pos,
                     __nv_bfloat16* __restrict__ dY, float* __restrict__ dw, int max_rows, int n, int d, int k, int B,
                     int C) {
  constexpr int U = 4;
  const int live_rows = min(meta[1], max_rows);
  const int vec = d / 8;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < live_rows; row += warps) {
    const int a = row_src[row];
    uint4* orow = reinterpret_cast<uint4*>(dY + (size_t)row * d);
    float dot = 0.f;
    if (a < 0) {
      for (int v = lane; v < vec; v += 32) orow[v] = make_uint4(0, 0, 0, 0);
    } else {
      const uint4* grow = reinterpret_cast<const uint4*>(dout + (size_t)(a / k) * d);
      const uint4* yrow = reinterpret_cast<const uint4*>(Y + (size_t)row * d);
      const float s = w[a];
      for (int v0 = lane; v0 < vec; v0 += 32 * U) {
        uint4 g[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int v = v0 + u * 32;
          g[u] = v < vec ? __ldg(grow + v) : make_uint4(0, 0, 0, 0);
          y[u] = v < vec ? __ldg(yrow + v) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int v = v0 + u * 32;
          if (v >= vec) break;
          __nv_bfloat162* q1 = reinterpret_cast<__nv_bfloat162*>(&g[u]);
          const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&y[u]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(q1[i]), h = __bfloat1622float2(q2[i]);
            dot += f.x * h.x + f.y * h.y;
            q1[i] = __floats2bfloat162_rn(f.x * s, f.y * s);
          }
          orow[v] = g[u];
        }
      }
      dot = warp_sum(dot);
    }
    if (lane == 0) {
      if (C > 0) {
        const int e = row / (B * C), b = row / C - e * B;
        dw[((size_t)b * k + e) * C + row % C] = dot;
      } else if (a >= 0) {
        dw[a] = dot;
      }
    }
  }
  if (C == 0)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
      if (pos[i] < 0) dw[i] = 0.f;
}

// Expert choice in the bookkeeping of token choice with k = E: row (e, b, c) holds token b * S + tok[b][e][c] of the T
// tokens.  row_src[row] = assignment t * E + e, pos[assignment] = row (preset to -1), weight[assignment] = wts[b][e][c];
// the weights of assignments without a row are never read.  A token outside [0, S) leaves its row empty and sets status
// 310.  One launch in place of a dozen elementwise and indexing ones.
__global__ void moe_choice_plan_kernel(const long long* __restrict__ tok, const float* __restrict__ wts,
                                       int* __restrict__ row_src, int* __restrict__ pos, float* __restrict__ weight,
                                       int* __restrict__ meta, int B, int E, int C, int S, int* __restrict__ status) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row < 2) meta[row] = E * B * C;
  if (row >= E * B * C) return;
  const int e = row / (B * C), b = row / C - e * B, c = row % C;
  const size_t src = ((size_t)b * E + e) * C + c;
  const long long t = tok[src];
  if (t < 0 || t >= S) {
    row_src[row] = -1;
    atomicExch(status, 310);
    return;
  }
  const int a = ((int)t + b * S) * E + e;
  row_src[row] = a;
  pos[a] = row;
  weight[a] = wts[src];
}

// dw[t,k] = <dout[t], Y[pos[t,k]]>.  One warp per assignment.
__global__ void moe_combine_dw_kernel(const __nv_bfloat16* __restrict__ Y, const __nv_bfloat16* __restrict__ dout,
                                      const int* __restrict__ pos, float* __restrict__ dw, int n, int k, int d) {
  const int vec = d / 8;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (int a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; a < n; a += warps) {
    const int p = pos[a];
    float s = 0.f;
    if (p >= 0) {
      const uint4* yr = reinterpret_cast<const uint4*>(Y + (size_t)p * d);
      const uint4* gr = reinterpret_cast<const uint4*>(dout + (size_t)(a / k) * d);
      for (int v = lane; v < vec; v += 32) {
        uint4 r1 = yr[v], r2 = gr[v];
        const __nv_bfloat162* q1 = reinterpret_cast<const __nv_bfloat162*>(&r1);
        const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&r2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 f1 = __bfloat1622float2(q1[i]), f2 = __bfloat1622float2(q2[i]);
          s += f1.x * f2.x + f1.y * f2.y;
        }
      }
    }
    s = warp_sum(s);
    if (lane == 0) dw[a] = s;
  }
}

}  // namespace kmoe

using namespace kmoe;

extern "C" int kmoe_moe_max_rows(int n_assign, int E) {
  const int r = n_assign + E * (ROW_TILE - 1);
  return (r + ROW_TILE - 1) / ROW_TILE * ROW_TILE;
}

extern "C" int kmoe_moe_plan(const long long* idx, const unsigned char* keep, int n, int E, int max_rows,
                             int expert_base, int* pos, int* row_src, int* counts, int* offsets, int* tile_group,
                             int* meta, cudaStream_t st) {
  const size_t smem = ((size_t)PLAN_WARPS * E + E + 1) * sizeof(int);
  if (smem > 200 * 1024 || E >= 0xffff) return -1;
  static SmemLimit limit;
  if (smem > 48 * 1024 && !limit.raise(moe_plan_kernel, smem)) return -3;
  moe_plan_kernel<<<1, 32 * PLAN_WARPS, smem, st>>>(idx, keep, n, E, max_rows, expert_base, pos, row_src, counts, offsets,
                                                    tile_group, meta);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_moe_capacity_mask(const long long* idx, int n, int E, int cap, unsigned char* keep,
                                      cudaStream_t st) {
  const size_t smem = (size_t)PLAN_THREADS * E * sizeof(int);
  if (smem > 200 * 1024) return -1;
  static SmemLimit limit;
  if (smem > 48 * 1024 && !limit.raise(moe_capacity_mask_kernel, smem)) return -3;
  moe_capacity_mask_kernel<<<1, PLAN_THREADS, smem, st>>>(idx, n, E, cap, keep);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// `counts` holds k + 1 rows of E ints, zeroed by the caller: row j = expert loads at the start of slot j.
extern "C" int kmoe_moe_balanced_assign(const float* probs, unsigned char* taken, int* counts, long long* sel, int T,
                                        int E, int k, int cap, cudaStream_t st) {
  for (int j = 0; j < k; ++j) {
    if (j > 0) cudaMemcpyAsync(counts + (size_t)(j + 1) * E, counts + (size_t)j * E, E * sizeof(int),
                               cudaMemcpyDeviceToDevice, st);
    // slot j reads row j and accumulates the loads after the slot into row j + 1 (which starts as a copy of row j)
    moe_balanced_slot_kernel<<<148 * 4, 256, 0, st>>>(probs, taken, counts + (size_t)j * E,
                                                      counts + (size_t)(j + 1) * E, sel + j, k, T, E, cap);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_moe_gather_rows(const void* src, const int* row_src, const int* meta, void* dst, int max_rows, int d,
                                    int div, cudaStream_t st) {
  if (d % 8) return -1;
  moe_gather_rows_kernel<<<148 * 4, 256, 0, st>>>((const __nv_bfloat16*)src, row_src, meta, (__nv_bfloat16*)dst, max_rows,
                                                  d, div);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_moe_combine(const void* Y, const int* pos, const float* w, void* out, int T, int k, int d,
                                cudaStream_t st) {
  if (d % 8) return -1;
  if (T <= 0) return 0;
  const long long units = (long long)T * ((d / 8 + 63) / 64);
  const int grid = (int)((units + 7) / 8 < 148 * 8 ? (units + 7) / 8 : 148 * 8);
  moe_combine_kernel<<<grid, 256, 0, st>>>((const __nv_bfloat16*)Y, pos, w, (__nv_bfloat16*)out, T, k, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_moe_gather_dw(const void* dout, const int* row_src, const float* w, const void* Y, const int* meta,
                                  const int* pos, void* dY, float* dw, int max_rows, int n, int d, int k, int B, int C,
                                  cudaStream_t st) {
  if (d % 8 || k < 1 || (C == 0 && pos == nullptr)) return -1;
  if (max_rows <= 0) return 0;
  const int grid = (max_rows + 7) / 8;
  moe_gather_dw_kernel<<<grid < 148 * 8 ? grid : 148 * 8, 256, 0, st>>>((const __nv_bfloat16*)dout, row_src, w,
                                                                        (const __nv_bfloat16*)Y, meta, pos,
                                                                        (__nv_bfloat16*)dY, dw, max_rows, n, d, k, B, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_moe_choice_plan(const long long* tok, const float* wts, int* row_src, int* pos, float* weight,
                                    int* meta, int B, int E, int C, int S, int T, int* status, cudaStream_t st) {
  if ((long long)B * S != T) return -3;
  if ((long long)T * E > 0x7fffffff || (long long)B * E * C > 0x7fffff00) return -1;
  if (cudaMemsetAsync(pos, 0xff, (size_t)T * E * sizeof(int), st) != cudaSuccess) return -2;
  const int rows = B * E * C;
  moe_choice_plan_kernel<<<(rows + 255) / 256, 256, 0, st>>>(tok, wts, row_src, pos, weight, meta, B, E, C, S, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int kmoe_moe_combine_dw(const void* Y, const void* dout, const int* pos, float* dw, int n, int k, int d,
                                   cudaStream_t st) {
  if (d % 8) return -1;
  moe_combine_dw_kernel<<<148 * 4, 256, 0, st>>>((const __nv_bfloat16*)Y, (const __nv_bfloat16*)dout, pos, dw, n, k,
                                                 d);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
