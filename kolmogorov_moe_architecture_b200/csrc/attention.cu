// Causal grouped-query flash attention for sm_100a: tcgen05 MMAs with TMEM accumulators,
// TMA-fed 128B-swizzled shared memory, online softmax in registers.
//
// Layouts: q, o, do, dq [B, S, H, D]; k, v, dk, dv [B, S, Hkv, D] (bf16, contiguous);
// lse [B, H, S] fp32 (natural log).  Query head h reads KV head h / (H / Hkv) directly -
// K and V are never expanded to H heads.
//
// head_dim 64 and 128, 320-thread CTAs - eight softmax warps in two warpgroups, a TMA producer warp, an MMA warp - and
// 128-key / 128-query steps.
//   forward   attn_fwd2_kernel: one or two 128-query tiles per CTA, one per warpgroup; S = Q K^T in TMEM, the score row
//             is read into registers once, P is written as packed bf16 over the S columns and feeds O += P V as
//             the A operand from tensor memory; O stays in TMEM and is rescaled only when the row maximum grew by
//             more than 2^8.
//   backward  attn_stats_kernel (row statistics), attn_bwd_dq2_kernel (loop over key blocks of a query block) and
//             attn_bwd_dkv2_kernel (loop over the query heads of the group and their query blocks for a key block);
//             both recompute P from the saved lse (no atomics, deterministic); the warpgroups split the 128 columns of
//             an accumulator in halves; P^T / dS^T / dS are packed over consumed accumulator columns and enter the next
//             MMA from tensor memory.
// The tile index is the slowest grid dimension, so the heavy tiles of all heads run first.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <cstdlib>

#include <mutex>

#include "kmoe_api.h"
#include "ptx.cuh"
#include "tmap_host.h"

namespace kmoe {

constexpr int ATT_BLK = 128;             // query rows per CTA and keys per step
constexpr int PANEL_BYTES = ATT_BLK * 128;  // one 64-column bf16 panel of a 128-row tile

struct AttnArgs {
  int B, S, H, Hkv;
  float scale_log2;  // softmax scale * log2(e)
  __nv_bfloat16* out;
  float* lse;
  int* status;
  // optional (B, S): first position of the packed document that contains each position; a query then sees
  // only keys k with doc_start[q] <= k <= q (block-diagonal causal mask of packed sequences)
  const int* doc_start;
  int q_tiles;       // forward: 128-query tiles per CTA, 1 or 2
};

constexpr float RESCALE_THRESHOLD = 8.0f;          // log2 units: rescale O only when the row max grew by > 2^8

// ------------------------------------------------------------ forward, two query tiles per CTA
// One CTA per SM owns 256 query rows as two 128-row tiles (or 128 rows as one, where the grid is small), each with its
// own softmax warpgroup, S and O accumulators (4 x 128 TMEM columns in all) and barriers; both tiles share the K/V tiles of a 128-key step.
//   warps 0-3 / 4-7  softmax of tile 0 / 1 (thread = query row)
//   warp 8           TMA producer: Q tiles once, K_j / V_j into 2-stage rings
//   warp 9           MMA issuer: S_t = Q_t K_j^T (128 x 128 x 128), O_t += P_t V_j with P_t read from TMEM
// P is written as packed bf16 over the first 64 columns of the tile's own S accumulator (the softmax has the whole
// 128-value score row in registers by then), so no shared memory is spent on P and the PV MMA takes its A operand
// from tensor memory.  The tensor pipe executes one tile's MMAs while the
// other tile's warpgroup is in its softmax; 128-key steps halve the number of barrier round trips per key.
constexpr int F2_KEYS = 128;
constexpr int F2_THREADS = 320;

// 2^x on the FMA pipe (x <= ~10): round-to-nearest split x = n + f, f in [-0.5, 0.5], cubic for 2^f, exponent
// added in integer.  Relative error ~1e-4, far below the bf16 rounding of P.  Used for a share of the
// exponentials of 128-wide heads so that the MUFU pipe (16 per clock and SM) is not the only limit of the softmax.  64-wide
// heads take MUFU alone: with the share their saved row sums were off by up to 2e-4 (now 1e-6); 4x2048x16 78.0 -> 80.7 us,
// 8x1021x12 43.3 -> 43.5 us.
__device__ __forceinline__ float ex2_fma(float x) {
  x = fmaxf(x, -125.f);
  const float t = x + 12582912.f;                   // 1.5 * 2^23: the integer part lands in the low mantissa bits
  const float f = x - (t - 12582912.f);
  float p = 0.0555041f;
  p = fmaf(p, f, 0.2402265f);
  p = fmaf(p, f, 0.6931472f);
  p = fmaf(p, f, 1.0f);
  return __int_as_float(__float_as_int(p) + (__float_as_int(t) << 23));
}

template <int D>
__global__ void __launch_bounds__(F2_THREADS, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const AttnArgs a) {
  static_assert(D == 64 || D == 128, "head_dim is one or two 64-column panels");
  constexpr int NP = D / 64;
  constexpr int TILE_BYTES = NP * PANEL_BYTES;       // 128 rows x D bf16 columns in 64-column panels
  constexpr uint32_t IDESC_S = make_idesc_f16(128, F2_KEYS, 1, KMOE_MAJOR_K, KMOE_MAJOR_K);
  constexpr uint32_t IDESC_PV = make_idesc_f16(128, D, 1, KMOE_MAJOR_K, KMOE_MAJOR_MN);
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t COL_S = 0, COL_O = 256;          // S_t at COL_S + 128 t, O_t at COL_O + 128 t

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                           // 2 tiles
  uint8_t* sK = sQ + 2 * TILE_BYTES;         // 2 stages
  uint8_t* sV = sK + 2 * TILE_BYTES;         // 2 stages
  __shared__ uint64_t q_full, k_full[2], v_full[2], k_empty[2], v_empty[2], s_full[2], p_full[2], pv_done[2];
  __shared__ uint32_t tmem_slot;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the block index is the slowest grid dimension: all heavy (late) query blocks are scheduled before any lighter one
  const int qb = gridDim.z - 1 - blockIdx.z;
  const int h = blockIdx.x, b = blockIdx.y;
  const int hkv = h / (a.H / a.Hkv);
  const int q0 = qb * 128 * a.q_tiles;
  // packed documents: key blocks that end before the document of the CTA's first query are invisible to all rows
  const int jlo = a.doc_start != nullptr ? a.doc_start[(size_t)b * a.S + q0] / F2_KEYS : 0;
  // visited key blocks per tile (causal): tile t sees keys < min(q0 + 128 (t + 1), S)
  int nb[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int kmax = min(q0 + 128 * (t + 1), a.S);
    nb[t] = (t < a.q_tiles && q0 + 128 * t < a.S) ? max((kmax + F2_KEYS - 1) / F2_KEYS - jlo, 0) : 0;
  }
  const int nblk = max(nb[0], nb[1]);

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&v_full[i], 1);
      mbar_init(&k_empty[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 128); mbar_init(&pv_done[i], 1);
    }
    mbar_fence_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV);
  }
  if (warp == 9) {
    tmem_alloc(&tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one() && nblk > 0) {
      mbar_expect_tx(&q_full, a.q_tiles * TILE_BYTES);
      for (int t = 0; t < a.q_tiles; ++t)
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sQ + t * TILE_BYTES + p * PANEL_BYTES, &tmQ, &q_full, p * 64, h, q0 + t * 128, b);
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1;
        const uint32_t par = ((j >> 1) & 1) ^ 1;
        if (!mbar_wait(&k_empty[st], par)) { atomicExch(a.status, 31); goto teardown; }
        mbar_expect_tx(&k_full[st], TILE_BYTES);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sK + st * TILE_BYTES + p * PANEL_BYTES, &tmK, &k_full[st], p * 64, hkv, (jlo + j) * F2_KEYS, b);
        if (!mbar_wait(&v_empty[st], par)) { atomicExch(a.status, 32); goto teardown; }
        mbar_expect_tx(&v_full[st], TILE_BYTES);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sV + st * TILE_BYTES + p * PANEL_BYTES, &tmV, &v_full[st], p * 64, hkv, (jlo + j) * F2_KEYS, b);
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one() && nblk > 0) {
      auto issue_S = [&](int t, int j) {
        const uint32_t qa = smem_u32(sQ + t * TILE_BYTES), ka = smem_u32(sK + (j & 1) * TILE_BYTES);
#pragma unroll
        for (int k4 = 0; k4 < D / 16; ++k4) {
          const uint32_t off = (k4 >> 2) * PANEL_BYTES + (k4 & 3) * 32;
          umma_f16(tmem + COL_S + t * 128, make_smem_desc_sw128(qa + off, 16, 1024),
                   make_smem_desc_sw128(ka + off, 16, 1024), IDESC_S, k4 > 0);
        }
        umma_commit(&s_full[t]);
      };
      if (!mbar_wait(&q_full, 0)) { atomicExch(a.status, 33); goto teardown; }
      if (!mbar_wait(&k_full[0], 0)) { atomicExch(a.status, 34); goto teardown; }
      tc_fence_after();
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (nb[t] > 0) issue_S(t, 0);
      umma_commit(&k_empty[0]);
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1;
        if (!mbar_wait(&v_full[st], (j >> 1) & 1)) { atomicExch(a.status, 35); goto teardown; }
        if (j + 1 < nblk && !mbar_wait(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1)) {
          atomicExch(a.status, 36);
          goto teardown;
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j >= nb[t]) continue;
          if (!mbar_wait(&p_full[t], j & 1)) { atomicExch(a.status, 37); goto teardown; }
          tc_fence_after();
          const uint32_t va = smem_u32(sV + st * TILE_BYTES);
#pragma unroll
          for (int k4 = 0; k4 < F2_KEYS / 16; ++k4)   // A = P_t from tensor memory: 16 keys = 8 packed columns
            umma_f16_ts(tmem + COL_O + t * 128, tmem + COL_S + t * 128 + k4 * 8,
                        make_smem_desc_sw128(va + k4 * 16 * 128, PANEL_BYTES, 1024), IDESC_PV, (j > 0 || k4 > 0));
          umma_commit(&pv_done[t]);
          if (j + 1 < nb[t]) issue_S(t, j + 1);       // overwrites S_t / P_t: ordered behind the PV just issued
        }
        if (j + 1 < nblk) umma_commit(&k_empty[(j + 1) & 1]);
        umma_commit(&v_empty[st]);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    const int t = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const int qt0 = q0 + t * 128;                 // first query row of this tile
    const int qi = qt0 + r;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t ts = tmem + lane_base + COL_S + t * 128;
    const uint32_t to = tmem + lane_base + COL_O + t * 128;
    float m_used = -INFINITY, l = 0.f;
    const int qstart = (a.doc_start != nullptr && qi < a.S) ? a.doc_start[(size_t)b * a.S + qi] : 0;
    const float sc = a.scale_log2;
    for (int j = 0; j < nb[t]; ++j) {
      if (!mbar_wait(&s_full[t], j & 1)) { if (lane == 0) atomicExch(a.status, 38); goto teardown; }
      tc_fence_after();
      const int k0 = (jlo + j) * F2_KEYS;
      const bool need_mask = (k0 + F2_KEYS > qt0) || (k0 + F2_KEYS > a.S) || (k0 < qstart);
      // The whole row of scores (128 values) is read into registers once; the mask is applied in a separate,
      // rarely taken branch.
      uint32_t v[F2_KEYS];
#pragma unroll
      for (int c = 0; c < F2_KEYS; c += 32) tmem_ld_32x32(ts + c, *reinterpret_cast<uint32_t(*)[32]>(&v[c]));
      tmem_ld_wait();
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < F2_KEYS; ++i) {
          const int kk = k0 + i;
          if (kk > qi || kk >= a.S || kk < qstart) v[i] = 0xff800000u;      // -inf
        }
      }
      float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
      for (int i = 0; i < F2_KEYS; i += 4) {
        m0 = fmaxf(m0, __uint_as_float(v[i]));
        m1 = fmaxf(m1, __uint_as_float(v[i + 1]));
        m2 = fmaxf(m2, __uint_as_float(v[i + 2]));
        m3 = fmaxf(m3, __uint_as_float(v[i + 3]));
      }
      const float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * sc;      // scale > 0: max of the scaled scores
      const bool grow = mx > m_used + RESCALE_THRESHOLD;      // always true on the first step
      const float m_new = grow ? mx : m_used;
      const float alpha = grow ? exp2f(m_used - m_new) : 1.f;
      const float m_exp = (m_new == -INFINITY) ? 0.f : m_new;   // rows that have not met a visible key yet
      if (j > 0 && __any_sync(0xffffffffu, grow)) {
        // s_full for step j was committed after PV of step j-1 in the same in-order pipe: O is at rest
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32(to + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(to + c, o);
        }
        tmem_st_wait();
      }
      // p = 2^(s * scale - m), packed bf16 written over the first 64 columns of S (all of S is in registers)
      const uint64_t sc2 = pack_f32x2(sc, sc), nm2 = pack_f32x2(-m_exp, -m_exp);
      uint64_t rsum = pack_f32x2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < F2_KEYS; c += 32) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float x0, x1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[c + i]), __uint_as_float(v[c + i + 1])), sc2, nm2), x0, x1);
          // head_dim 128: every fourth pair on the FMA pipe, the rest on MUFU
          const float p0 = (D == 128 && (i & 6) == 6) ? ex2_fma(x0) : ex2_approx(x0);
          const float p1 = (D == 128 && (i & 6) == 6) ? ex2_fma(x1) : ex2_approx(x1);
          rsum = add_f32x2(rsum, pack_f32x2(p0, p1));
          pk[i >> 1] = pack_bf16(p0, p1);
        }
        tmem_st_32x16(ts + (c >> 1), pk);
      }
      float rs0, rs1;
      unpack_f32x2(rsum, rs0, rs1);
      const float rs = rs0 + rs1;
      tmem_st_wait();
      l = l * alpha + rs;
      m_used = m_new;
      tc_fence_before();
      mbar_arrive(&p_full[t]);
    }
    if (nb[t] > 0) {
      if (!mbar_wait(&pv_done[t], (nb[t] - 1) & 1)) { if (lane == 0) atomicExch(a.status, 39); goto teardown; }
      tc_fence_after();
      const bool row_ok = qi < a.S;
      const float inv = 1.f / l;
      __nv_bfloat16* orow = a.out + (((size_t)b * a.S + (row_ok ? qi : 0)) * a.H + h) * D;
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(to + c, v);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            *reinterpret_cast<uint4*>(orow + c + i) =
                make_uint4(pack_bf16(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv),
                           pack_bf16(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv),
                           pack_bf16(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv),
                           pack_bf16(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv));
        }
      }
      if (row_ok) a.lse[((size_t)b * a.H + h) * a.S + qi] = (m_used + log2f(l)) * 0.6931471805599453f;
      tc_fence_before();
    }
  }

teardown:
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

}  // namespace kmoe

// ------------------------------------------------------------------- backward
namespace kmoe {

struct AttnBwdArgs {
  int B, S, H, Hkv;
  float scale, scale_log2;
  int Sp;               // S rounded up to whole 128-row blocks: pitch of the row statistics
  const float* nlse;    // [B,H,Sp]  -lse * log2(e): the exponent of P is s * scale_log2 + this
  const float* ndelta;  // [B,H,Sp]  -rowsum(dO * O) * scale: dS = P * (dP * scale + this)
  __nv_bfloat16* dq;    // [B,S,H,D]
  __nv_bfloat16* dk;    // [B,S,Hkv,D]
  __nv_bfloat16* dv;
  int* status;
  const int* doc_start;  // optional (B, S), see AttnArgs
};

// Row statistics of the backward pass, in the form and place its kernels want them: one row of Sp = whole 128-row
// blocks per (b, h), so that a block's 128 values are one aligned 512-byte bulk copy; positions past S hold zeros.
//   nlse = -lse * log2(e),  ndelta = -scale * sum_d dO * O
// D / 8 lanes per (b, s, h) row (one 16-byte vector of each operand per lane) and four rows per lane in flight: the
// kernel only has to keep enough loads outstanding to stream O and dO once.  B = 4, S = 2048, 16 x 128: 34.3 us with one
// row per warp and pass (half of the lanes without work), 17.1 us this way, 10.3 us at the copy rate.
template <int D>
__global__ void __launch_bounds__(256) attn_stats_kernel(const __nv_bfloat16* __restrict__ o,
                                                         const __nv_bfloat16* __restrict__ d_o,
                                                         const float* __restrict__ lse, float* __restrict__ nlse,
                                                         float* __restrict__ ndelta, long long rows, int S, int Sp, int H,
                                                         float scale) {
  constexpr int LPR = D / 8, RPB = 256 / LPR, U = 4;
  const int sub = threadIdx.x % LPR, r_in = threadIdx.x / LPR;
  const long long row0 = (long long)blockIdx.x * (RPB * U) + r_in;      // rows of the padded (B, Sp, H)
  uint4 x[U], y[U];
  long long at[U];        // place in [B, H, Sp]
  float ls[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long row = row0 + u * RPB;
    const int h = (int)(row % H);
    const long long bs = row / H;
    const int s_ = (int)(bs % Sp);
    const long long b = bs / Sp;
    const bool ok = row < rows && s_ < S;
    const long long src = ((b * S + s_) * H + h) * D;
    x[u] = ok ? __ldg(reinterpret_cast<const uint4*>(o + src) + sub) : make_uint4(0, 0, 0, 0);
    y[u] = ok ? __ldg(reinterpret_cast<const uint4*>(d_o + src) + sub) : make_uint4(0, 0, 0, 0);
    at[u] = row < rows ? (b * H + h) * Sp + s_ : -1;
    ls[u] = (ok && sub == 0) ? __ldg(lse + (b * H + h) * S + s_) : 0.f;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const __nv_bfloat162* p1 = reinterpret_cast<const __nv_bfloat162*>(&x[u]);
    const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&y[u]);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f1 = __bfloat1622float2(p1[i]), f2 = __bfloat1622float2(p2[i]);
      acc += f1.x * f2.x + f1.y * f2.y;
    }
#pragma unroll
    for (int k = LPR / 2; k > 0; k >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, k);
    if (sub == 0 && at[u] >= 0) {
      nlse[at[u]] = -ls[u] * 1.4426950408889634f;
      ndelta[at[u]] = -acc * scale;
    }
  }
}

// ------------------------------------------------- backward: 128 x 128 steps, P and dS in TMEM
// Both kernels below keep the structure of the two-tile forward: 8 softmax warps (two warpgroups that split the
// 128 columns of an accumulator in halves; thread = accumulator row), warp 8 is the TMA producer, warp 9 issues
// the MMAs.  The bf16 operands made by the threads (P^T and dS^T for dK/dV, dS for dQ) are written as packed
// pairs over accumulator columns the same warpgroup has already consumed and enter the next MMA as its A
// operand from tensor memory, so no shared memory and no proxy fence is spent on them.  The work of a step is
// two chains that the tensor pipe interleaves: S -> P (exponentials) and dP -> dS (needs P, kept in
// registers); while the threads are in one chain the pipe executes the MMAs of the other.
constexpr int B2_THREADS = 320;
constexpr int DKV2_Q_STAGES = 3;
// Shared memory of the dK/dV kernel: K, V, three Q and two dO tiles, the row statistics and the barriers.  At head_dim
// 128 this is all of an SM's 227 KB but 400 bytes, so the dynamic segment (there is no static one) must start on a 1 KB
// boundary by itself; the kernel checks that.
template <int D>
constexpr int dkv2_smem_bytes() { return 7 * (D / 64) * PANEL_BYTES + 5 * 512 + 256; }

// dK, dV of one (128-key block, KV head, batch): loops over the query heads of the group and over the
// 128-query blocks at or after the key block.  TMEM: S^T | dP^T | dV | dK, 128 columns each.
//
// The loads of a step (Q and its ndelta, dO and its nlse) are TMA / bulk copies issued by one thread.  Q is held until
// the dK MMAs, the last of a step: with two stages (and the statistics loaded by the producer warp itself) the loads of
// step i + 2 started a load latency before their use, which cost 0.3 us
// per step (4x2048x16/4: 142 -> 123 us).
//
// The key blocks of a KV head are few when the batch is small, and the first of them visits every query block of every
// head of the group.  A cluster of `split` CTAs shares a key block then, each taking 1 / split of the group's heads;
// the partial sums meet in shared memory (fp32, fixed order) and each CTA stores its share of the rows.
template <int D>
__global__ void __launch_bounds__(B2_THREADS, 1)
attn_bwd_dkv2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const AttnBwdArgs a, const int split) {
  constexpr int NP = D / 64;
  constexpr int TILE_BYTES = NP * PANEL_BYTES;       // 128 rows x D bf16 columns
  constexpr int NQ = DKV2_Q_STAGES;
  constexpr uint32_t IDESC_ST = make_idesc_f16(128, 128, 1, KMOE_MAJOR_K, KMOE_MAJOR_K);
  constexpr uint32_t IDESC_ACC = make_idesc_f16(128, D, 1, KMOE_MAJOR_K, KMOE_MAJOR_MN);
  constexpr uint32_t TMEM_COLS = 512, COL_ST = 0, COL_DPT = 128, COL_DV = 256, COL_DK = 384;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  uint8_t* sK = smem;
  uint8_t* sV = sK + TILE_BYTES;
  uint8_t* sQ = sV + TILE_BYTES;                 // NQ stages
  uint8_t* sdO = sQ + NQ * TILE_BYTES;           // 2 stages, released by the dV MMAs in mid-step
  float(*s_ndelta)[128] = reinterpret_cast<float(*)[128]>(sdO + 2 * TILE_BYTES);   // one row per Q stage
  float(*s_nlse)[128] = s_ndelta + NQ;                                             // one row per dO stage
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_nlse + 2);
  uint64_t &kv_full = bars[0], &st_full = bars[1], &dpt_full = bars[2], &p_full = bars[3], &ds_full = bars[4],
           &acc_full = bars[5];
  uint64_t *q_full = bars + 6, *q_empty = bars + 9, *do_full = bars + 12, *do_empty = bars + 14;
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 16);
  constexpr int PART_PITCH = 2 * D + 4;          // fp32 row of partial sums: conflict-free float4 rows

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (smem_u32(smem) & 1023u) {                  // never: see dkv2_smem_bytes
    if (threadIdx.x == 0) atomicExch(a.status, 61);
    return;
  }
  // the key block is the slowest grid dimension: the heavy (early) key blocks of all heads are scheduled first
  const int kb = blockIdx.z, hkv = blockIdx.x / split, part = blockIdx.x % split, b = blockIdx.y;
  const int G = a.H / a.Hkv / split;             // query heads of this CTA
  const int h0 = hkv * (a.H / a.Hkv) + part * G;
  const int k0 = kb * ATT_BLK;
  const int qblk1 = (a.S + ATT_BLK - 1) / ATT_BLK;
  int per_head = qblk1 - kb;
  if (a.doc_start != nullptr) {
    // packed documents: once a query block starts in a document that begins after this key block's last key,
    // it and all later query blocks cannot see the block (document starts do not decrease along the sequence)
    const int klast = min(k0 + ATT_BLK, a.S) - 1;
    for (int i = 1; i < per_head; ++i) {
      if (a.doc_start[(size_t)b * a.S + (kb + i) * ATT_BLK] > klast) { per_head = i; break; }
    }
  }
  const int niter = per_head * G;

  if (threadIdx.x == 0) {
    mbar_init(&kv_full, 1);
    for (int i = 0; i < NQ; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1); }
    mbar_init(&st_full, 1); mbar_init(&dpt_full, 1);
    mbar_init(&p_full, 256); mbar_init(&ds_full, 256); mbar_init(&acc_full, 1);
    mbar_fence_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmdO); prefetch_tmap(&tmK); prefetch_tmap(&tmV);
  }
  if (warp == 9) { tmem_alloc(&tmem_slot, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 8) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      auto load_q = [&](int it) {
        const int qs = it % NQ, h = h0 + it / per_head, qrow = (kb + it % per_head) * ATT_BLK;
        mbar_expect_tx(&q_full[qs], TILE_BYTES + 512);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sQ + qs * TILE_BYTES + p * PANEL_BYTES, &tmQ, &q_full[qs], p * 64, h, qrow, b);
        bulk_load(s_ndelta[qs], a.ndelta + ((size_t)b * a.H + h) * a.Sp + qrow, 512, &q_full[qs]);
      };
      auto load_do = [&](int it) {
        const int os = it & 1, h = h0 + it / per_head, qrow = (kb + it % per_head) * ATT_BLK;
        mbar_expect_tx(&do_full[os], TILE_BYTES + 512);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sdO + os * TILE_BYTES + p * PANEL_BYTES, &tmdO, &do_full[os], p * 64, h, qrow, b);
        bulk_load(s_nlse[os], a.nlse + ((size_t)b * a.H + h) * a.Sp + qrow, 512, &do_full[os]);
      };
      mbar_expect_tx(&kv_full, 2 * TILE_BYTES);
#pragma unroll
      for (int p = 0; p < NP; ++p) tma_load_4d(sK + p * PANEL_BYTES, &tmK, &kv_full, p * 64, hkv, k0, b);
      if (niter > 0) load_q(0);
#pragma unroll
      for (int p = 0; p < NP; ++p) tma_load_4d(sV + p * PANEL_BYTES, &tmV, &kv_full, p * 64, hkv, k0, b);
      if (niter > 0) load_do(0);
      for (int it = 1; it < niter; ++it) {
        // the Q stage is free once the dK MMAs of step it - 3 have completed, the dO stage once the dV MMAs of step
        // it - 2 have (those come first)
        if (!mbar_wait(&q_empty[it % NQ], ((it / NQ) & 1) ^ 1)) { atomicExch(a.status, 41); goto finish; }
        load_q(it);
        if (!mbar_wait(&do_empty[it & 1], ((it >> 1) & 1) ^ 1)) { atomicExch(a.status, 40); goto finish; }
        load_do(it);
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one() && niter > 0) {
      const uint32_t ka = smem_u32(sK), va = smem_u32(sV);
      // S^T = K Q^T or dP^T = V dO^T of one stage: 128 x 128 x 128
      auto issue_t = [&](uint32_t col, uint32_t a_base, uint32_t b_base) {
#pragma unroll
        for (int k4 = 0; k4 < D / 16; ++k4) {
          const uint32_t off = (k4 >> 2) * PANEL_BYTES + (k4 & 3) * 32;
          umma_f16(tmem + col, make_smem_desc_sw128(a_base + off, 16, 1024),
                   make_smem_desc_sw128(b_base + off, 16, 1024), IDESC_ST, k4 > 0);
        }
      };
      // acc += X^T Y with X^T (128 keys x 128 queries, packed bf16) in tensor memory: queries 0-63 sit in the
      // 32 columns at `col`, queries 64-127 in the 32 columns at `col` + 64 (each warpgroup packs over its own half)
      auto issue_acc = [&](uint32_t acc, uint32_t col, uint32_t y_base, bool first) {
#pragma unroll
        for (int k4 = 0; k4 < ATT_BLK / 16; ++k4)
          umma_f16_ts(tmem + acc, tmem + col + (k4 >> 2) * 64 + (k4 & 3) * 8,
                      make_smem_desc_sw128(y_base + k4 * 16 * 128, PANEL_BYTES, 1024), IDESC_ACC, (!first || k4 > 0));
      };
      if (!mbar_wait(&kv_full, 0)) { atomicExch(a.status, 42); goto finish; }
      if (!mbar_wait(&q_full[0], 0)) { atomicExch(a.status, 43); goto finish; }
      tc_fence_after();
      issue_t(COL_ST, ka, smem_u32(sQ));
      umma_commit(&st_full);
      if (!mbar_wait(&do_full[0], 0)) { atomicExch(a.status, 43); goto finish; }
      tc_fence_after();
      issue_t(COL_DPT, va, smem_u32(sdO));
      umma_commit(&dpt_full);
      for (int it = 0; it < niter; ++it) {
        const int qs = it % NQ, qn = (it + 1) % NQ, os = it & 1, on = os ^ 1;
        const uint32_t qa = smem_u32(sQ + qs * TILE_BYTES), da = smem_u32(sdO + os * TILE_BYTES);
        // chain 1: P^T(it) -> dV, then S^T(it + 1) over the same columns (in order behind the dV MMAs)
        if (!mbar_wait(&p_full, it & 1)) { atomicExch(a.status, 44); goto finish; }
        tc_fence_after();
        issue_acc(COL_DV, COL_ST, da, it == 0);
        umma_commit(&do_empty[os]);
        if (it + 1 < niter) {
          if (!mbar_wait(&q_full[qn], ((it + 1) / NQ) & 1)) { atomicExch(a.status, 45); goto finish; }
          tc_fence_after();
          issue_t(COL_ST, ka, smem_u32(sQ + qn * TILE_BYTES));
          umma_commit(&st_full);
        }
        // chain 2: dS^T(it) -> dK, then dP^T(it + 1)
        if (!mbar_wait(&ds_full, it & 1)) { atomicExch(a.status, 46); goto finish; }
        tc_fence_after();
        issue_acc(COL_DK, COL_DPT, qa, it == 0);
        umma_commit(&q_empty[qs]);
        if (it + 1 < niter) {
          if (!mbar_wait(&do_full[on], ((it + 1) >> 1) & 1)) { atomicExch(a.status, 45); goto finish; }
          tc_fence_after();
          issue_t(COL_DPT, va, smem_u32(sdO + on * TILE_BYTES));
          umma_commit(&dpt_full);
        }
      }
      umma_commit(&acc_full);
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups (thread = key row)
    const int wg = warp >> 2;
    const int cb = wg * 64;                        // this warpgroup's query columns of the step
    const int r = (warp & 3) * 32 + lane;
    const int kj = k0 + r;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem + lane_base + COL_ST + cb;
    const uint32_t t_dp = tmem + lane_base + COL_DPT + cb;
    const uint64_t sl2 = pack_f32x2(a.scale_log2, a.scale_log2), sc2 = pack_f32x2(a.scale, a.scale);
    // The queries that see key kj are [kj, vis_end): up to the sequence's end or, packed, to the first query whose
    // document starts behind the key (starts do not decrease, so a binary search finds it, once per CTA and under the
    // first loads; testing the start of every query of a step was 64 loads per thread and step, 8x1021x12/3x64 with
    // four documents 90 -> 57 us, 4x1024x12/3x128 without documents 43.7 -> 40.0).
    int vis_end = min(a.S, (kb + per_head) * ATT_BLK);
    if (a.doc_start != nullptr) {
      const int* ds = a.doc_start + (size_t)b * a.S;
      int lo = kj + 1;
      while (lo < vis_end) {
        const int mid = (lo + vis_end) >> 1;
        if (__ldg(ds + mid) > kj) vis_end = mid;
        else lo = mid + 1;
      }
    }
    if (kj >= a.S) vis_end = 0;
    const int warp_end = __shfl_sync(0xffffffffu, vis_end, 0);     // the smallest of the warp (or 0), as kj is lane's
    for (int it = 0; it < niter; ++it) {
      const int qs = it % NQ, os = it & 1;
      const int qrow = (kb + it % per_head) * ATT_BLK;
      if (!mbar_wait(&do_full[os], (it >> 1) & 1)) { if (lane == 0) atomicExch(a.status, 47); goto finish; }
      if (!mbar_wait(&st_full, it & 1)) { if (lane == 0) atomicExch(a.status, 48); goto finish; }
      tc_fence_after();
      // per-element tests only for steps that touch the diagonal, the sequence end or a document boundary
      const bool need_mask = (qrow < k0 + ATT_BLK) || (qrow + ATT_BLK > warp_end) || (k0 + ATT_BLK > a.S);
      uint64_t p2[32];                             // P of this thread's 64 queries, fp32 pairs
      {
        uint32_t sv[64];
        tmem_ld_32x32(t_s, *reinterpret_cast<uint32_t(*)[32]>(&sv[0]));
        tmem_ld_32x32(t_s + 32, *reinterpret_cast<uint32_t(*)[32]>(&sv[32]));
        tmem_ld_wait();
        if (need_mask) {
          const int first = kj - qrow - cb, end = vis_end - qrow - cb;
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (i < first || i >= end) sv[i] = 0xff800000u;          // p = 0
        }
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sl2,
                                       *reinterpret_cast<const uint64_t*>(&s_nlse[os][cb + 2 * i]));
          float x0, x1;
          unpack_f32x2(x, x0, x1);
          const float e0 = ex2_approx(x0), e1 = ex2_approx(x1);
          p2[i] = pack_f32x2(e0, e1);
          pk[i] = pack_bf16(e0, e1);
        }
        tmem_st_32x32(t_s, pk);                     // over columns this warpgroup has consumed
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full);
      if (!mbar_wait(&q_full[qs], (it / NQ) & 1)) { if (lane == 0) atomicExch(a.status, 47); goto finish; }
      if (!mbar_wait(&dpt_full, it & 1)) { if (lane == 0) atomicExch(a.status, 49); goto finish; }
      tc_fence_after();
      {
        uint32_t dv_[64];
        tmem_ld_32x32(t_dp, *reinterpret_cast<uint32_t(*)[32]>(&dv_[0]));
        tmem_ld_32x32(t_dp + 32, *reinterpret_cast<uint32_t(*)[32]>(&dv_[32]));
        tmem_ld_wait();
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          // dS = P * (dP - delta) * scale = P * (dP * scale - delta * scale)
          const uint64_t t = fma_f32x2(pack_f32x2(__uint_as_float(dv_[2 * i]), __uint_as_float(dv_[2 * i + 1])), sc2,
                                       *reinterpret_cast<const uint64_t*>(&s_ndelta[qs][cb + 2 * i]));
          float d0, d1;
          unpack_f32x2(mul_f32x2(p2[i], t), d0, d1);
          pk[i] = pack_bf16(d0, d1);
        }
        tmem_st_32x32(t_dp, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&ds_full);
    }
    if (niter > 0) {
      if (!mbar_wait(&acc_full, 0)) { if (lane == 0) atomicExch(a.status, 50); goto finish; }
      tc_fence_after();
    }
    if (split == 1) {
      const bool row_ok = kj < a.S;
      const size_t off = (((size_t)b * a.S + (row_ok ? kj : 0)) * a.Hkv + hkv) * D + wg * (D / 2);
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        __nv_bfloat16* drow = (which == 0 ? a.dv : a.dk) + off;
        const uint32_t col0 = (which == 0 ? COL_DV : COL_DK) + wg * (D / 2);
#pragma unroll 1
        for (int c = 0; c < D / 2; c += 32) {
          uint32_t v[32];
          if (niter > 0) {
            tmem_ld_32x32(tmem + lane_base + col0 + c, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8)
              *reinterpret_cast<uint4*>(drow + c + i) =
                  make_uint4(pack_bf16(__uint_as_float(v[i]), __uint_as_float(v[i + 1])),
                             pack_bf16(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])),
                             pack_bf16(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5])),
                             pack_bf16(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7])));
          }
        }
      }
    } else {
      // every MMA has completed and every load was consumed: the tiles' memory takes the fp32 rows [dV | dK]
      float* prow = reinterpret_cast<float*>(smem) + r * PART_PITCH + wg * (D / 2);
#pragma unroll
      for (int which = 0; which < 2; ++which) {
#pragma unroll 1
        for (int c = 0; c < D / 2; c += 32) {
          uint32_t v[32];
          if (niter > 0) {
            tmem_ld_32x32(tmem + lane_base + (which == 0 ? COL_DV : COL_DK) + wg * (D / 2) + c, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<uint4*>(prow + which * D + c + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
      }
    }
    tc_fence_before();
  }
finish:
  if (split > 1) {
    // also on the way out after a wait that ran out: the peers' memory must stay mapped until all have read it
    __syncthreads();
    __syncwarp();
    cluster_sync_all();
    const int rows = ATT_BLK / split;
    for (int i = threadIdx.x; i < rows * (2 * D / 8); i += B2_THREADS) {
      const int rr = part * rows + i / (2 * D / 8), c = (i % (2 * D / 8)) * 8;
      const float* mine = reinterpret_cast<const float*>(smem) + rr * PART_PITCH + c;
      float s8[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) s8[x] = 0.f;
      for (int p = 0; p < split; ++p) {
        const uint32_t addr = map_to_cta(mine, p);
        float4 v0 = ld_cluster_f4(addr), v1 = ld_cluster_f4(addr + 16);
        s8[0] += v0.x; s8[1] += v0.y; s8[2] += v0.z; s8[3] += v0.w;
        s8[4] += v1.x; s8[5] += v1.y; s8[6] += v1.z; s8[7] += v1.w;
      }
      if (k0 + rr < a.S) {
        __nv_bfloat16* dst = (c < D ? a.dv : a.dk) + (((size_t)b * a.S + k0 + rr) * a.Hkv + hkv) * D + (c % D);
        *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(s8[0], s8[1]), pack_bf16(s8[2], s8[3]),
                                                    pack_bf16(s8[4], s8[5]), pack_bf16(s8[6], s8[7]));
      }
    }
    __syncwarp();
    cluster_sync_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// dQ of one (128-query block, head, batch): loops over the 128-key blocks the block can see.
// TMEM: S | dP (two buffers, step parity) | dQ, 128 columns each.  S and dP of step j + 1 are issued as soon as
// the threads have read S of step j into registers, a whole thread phase ahead of their use.
template <int D>
__global__ void __launch_bounds__(B2_THREADS, 1)
attn_bwd_dq2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    const AttnBwdArgs a) {
  constexpr int NP = D / 64;
  constexpr int TILE_BYTES = NP * PANEL_BYTES;       // 128 rows x D bf16 columns
  constexpr uint32_t IDESC_S = make_idesc_f16(128, 128, 1, KMOE_MAJOR_K, KMOE_MAJOR_K);
  constexpr uint32_t IDESC_DQ = make_idesc_f16(128, D, 1, KMOE_MAJOR_K, KMOE_MAJOR_MN);
  constexpr uint32_t TMEM_COLS = 512, COL_S = 0, COL_DP = 128, COL_DQ = 384;   // dP buffer b at COL_DP + 128 b

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + TILE_BYTES;
  // K is held until the dQ MMAs of its step: a third stage lets the load of step j + 1 start a whole step ahead
  uint8_t* sK = sdO + TILE_BYTES;            // 3 stages
  uint8_t* sV = sK + 3 * TILE_BYTES;         // 2 stages
  __shared__ uint64_t qdo_full, k_full[3], v_full[2], k_empty[3], v_empty[2], s_full, s_free, dp_full[2], ds_full[2], dq_full;
  __shared__ uint32_t tmem_slot;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qb = gridDim.z - 1 - blockIdx.z;    // slowest grid dimension: heavy (late) query blocks first
  const int h = blockIdx.x, b = blockIdx.y;
  const int hkv = h / (a.H / a.Hkv);
  const int q0 = qb * ATT_BLK;
  const int kmax = min(q0 + ATT_BLK, a.S);
  // packed documents: key blocks that end before the document of the block's first query are invisible to all rows
  const int jlo = a.doc_start != nullptr ? a.doc_start[(size_t)b * a.S + q0] / ATT_BLK : 0;
  const int nblk = (kmax + ATT_BLK - 1) / ATT_BLK - jlo;

  if (threadIdx.x == 0) {
    mbar_init(&qdo_full, 1);
    for (int i = 0; i < 3; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); mbar_init(&dp_full[i], 1); mbar_init(&ds_full[i], 256);
    }
    mbar_init(&s_full, 1); mbar_init(&s_free, 256); mbar_init(&dq_full, 1);
    mbar_fence_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmdO); prefetch_tmap(&tmK); prefetch_tmap(&tmV);
  }
  if (warp == 9) { tmem_alloc(&tmem_slot, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 8) {
    if (elect_one() && nblk > 0) {
      mbar_expect_tx(&qdo_full, 2 * TILE_BYTES);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        tma_load_4d(sQ + p * PANEL_BYTES, &tmQ, &qdo_full, p * 64, h, q0, b);
        tma_load_4d(sdO + p * PANEL_BYTES, &tmdO, &qdo_full, p * 64, h, q0, b);
      }
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1, ks = j % 3;
        if (!mbar_wait(&k_empty[ks], ((j / 3) & 1) ^ 1)) { atomicExch(a.status, 51); goto teardown; }
        mbar_expect_tx(&k_full[ks], TILE_BYTES);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sK + ks * TILE_BYTES + p * PANEL_BYTES, &tmK, &k_full[ks], p * 64, hkv, (jlo + j) * ATT_BLK, b);
        if (!mbar_wait(&v_empty[st], ((j >> 1) & 1) ^ 1)) { atomicExch(a.status, 52); goto teardown; }
        mbar_expect_tx(&v_full[st], TILE_BYTES);
#pragma unroll
        for (int p = 0; p < NP; ++p)
          tma_load_4d(sV + st * TILE_BYTES + p * PANEL_BYTES, &tmV, &v_full[st], p * 64, hkv, (jlo + j) * ATT_BLK, b);
      }
    }
  } else if (warp == 9) {
    if (elect_one() && nblk > 0) {
      const uint32_t qa = smem_u32(sQ), da = smem_u32(sdO);
      auto issue_t = [&](uint32_t col, uint32_t a_base, uint32_t b_base) {
#pragma unroll
        for (int k4 = 0; k4 < D / 16; ++k4) {
          const uint32_t off = (k4 >> 2) * PANEL_BYTES + (k4 & 3) * 32;
          umma_f16(tmem + col, make_smem_desc_sw128(a_base + off, 16, 1024),
                   make_smem_desc_sw128(b_base + off, 16, 1024), IDESC_S, k4 > 0);
        }
      };
      if (!mbar_wait(&qdo_full, 0)) { atomicExch(a.status, 53); goto teardown; }
      if (!mbar_wait(&k_full[0], 0)) { atomicExch(a.status, 54); goto teardown; }
      tc_fence_after();
      issue_t(COL_S, qa, smem_u32(sK));
      umma_commit(&s_full);
      if (!mbar_wait(&v_full[0], 0)) { atomicExch(a.status, 55); goto teardown; }
      tc_fence_after();
      issue_t(COL_DP, da, smem_u32(sV));
      umma_commit(&dp_full[0]);
      umma_commit(&v_empty[0]);
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1, nx = st ^ 1, ks = j % 3, kn = (j + 1) % 3;
        if (j + 1 < nblk) {
          if (!mbar_wait(&k_full[kn], ((j + 1) / 3) & 1) || !mbar_wait(&v_full[nx], ((j + 1) >> 1) & 1)) {
            atomicExch(a.status, 54);
            goto teardown;
          }
          // S(j) is in the threads' registers: S(j + 1) may overwrite it.  dP(j + 1) goes to the other dP buffer,
          // whose dS(j - 1) the dQ MMAs of step j - 1 (earlier in this pipe) have consumed.
          if (!mbar_wait(&s_free, j & 1)) { atomicExch(a.status, 60); goto teardown; }
          tc_fence_after();
          issue_t(COL_S, qa, smem_u32(sK + kn * TILE_BYTES));
          umma_commit(&s_full);
          issue_t(COL_DP + nx * 128, da, smem_u32(sV + nx * TILE_BYTES));
          umma_commit(&dp_full[nx]);
          umma_commit(&v_empty[nx]);
        }
        // one barrier per dP buffer: a thread may finish dS(j + 1) (it needs only s_free of step j, not this
        // step's dQ MMAs) before a slower thread has arrived for dS(j), and the two must not share a phase
        if (!mbar_wait(&ds_full[st], (j >> 1) & 1)) { atomicExch(a.status, 56); goto teardown; }
        tc_fence_after();
        // dQ += dS K_j with dS (128 queries x 128 keys, packed bf16) in the step's dP buffer: keys 0-63 in its
        // first 32 columns, keys 64-127 in the 32 columns from column 64
        const uint32_t ka = smem_u32(sK + ks * TILE_BYTES);
#pragma unroll
        for (int k4 = 0; k4 < ATT_BLK / 16; ++k4)
          umma_f16_ts(tmem + COL_DQ, tmem + COL_DP + st * 128 + (k4 >> 2) * 64 + (k4 & 3) * 8,
                      make_smem_desc_sw128(ka + k4 * 16 * 128, PANEL_BYTES, 1024), IDESC_DQ, (j > 0 || k4 > 0));
        umma_commit(&k_empty[ks]);
      }
      umma_commit(&dq_full);
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups (thread = query row)
    const int wg = warp >> 2;
    const int cb = wg * 64;                        // this warpgroup's key columns of the step
    const int r = (warp & 3) * 32 + lane;
    const int qi = q0 + r;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const bool row_ok = qi < a.S;
    const size_t stat = ((size_t)b * a.H + h) * a.Sp + qi;          // qi < Sp always
    const float nl = a.nlse[stat], nd = a.ndelta[stat];
    const int qstart = (a.doc_start != nullptr && row_ok) ? a.doc_start[(size_t)b * a.S + qi] : 0;
    const uint32_t t_s = tmem + lane_base + COL_S + cb;
    const uint64_t sl2 = pack_f32x2(a.scale_log2, a.scale_log2), nlse = pack_f32x2(nl, nl);
    const uint64_t sc2 = pack_f32x2(a.scale, a.scale), nds = pack_f32x2(nd, nd);
    for (int j = 0; j < nblk; ++j) {
      if (!mbar_wait(&s_full, j & 1)) { if (lane == 0) atomicExch(a.status, 57); goto teardown; }
      tc_fence_after();
      const uint32_t t_dp = tmem + lane_base + COL_DP + (j & 1) * 128 + cb;
      const int k0 = (jlo + j) * ATT_BLK;
      const bool need_mask = (k0 + ATT_BLK > q0) || (k0 + ATT_BLK > a.S) || (k0 < qstart) || !row_ok;
      uint64_t p2[32];                             // P of this thread's 64 keys, fp32 pairs
      {
        uint32_t sv[64];
        tmem_ld_32x32(t_s, *reinterpret_cast<uint32_t(*)[32]>(&sv[0]));
        tmem_ld_32x32(t_s + 32, *reinterpret_cast<uint32_t(*)[32]>(&sv[32]));
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(&s_free);                      // S is in registers: the next S may be issued
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            const int kj = k0 + cb + i;
            if ((kj > qi) || (kj >= a.S) || !row_ok || (kj < qstart)) sv[i] = 0xff800000u;   // -inf: p = 0
          }
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float x0, x1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sl2, nlse),
                       x0, x1);
          p2[i] = pack_f32x2(ex2_approx(x0), ex2_approx(x1));
        }
      }
      if (!mbar_wait(&dp_full[j & 1], (j >> 1) & 1)) { if (lane == 0) atomicExch(a.status, 58); goto teardown; }
      tc_fence_after();
      {
        uint32_t dv_[64];
        tmem_ld_32x32(t_dp, *reinterpret_cast<uint32_t(*)[32]>(&dv_[0]));
        tmem_ld_32x32(t_dp + 32, *reinterpret_cast<uint32_t(*)[32]>(&dv_[32]));
        tmem_ld_wait();
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          // dS = P * (dP - delta) * scale = P * (dP * scale - delta * scale)
          const uint64_t t =
              fma_f32x2(pack_f32x2(__uint_as_float(dv_[2 * i]), __uint_as_float(dv_[2 * i + 1])), sc2, nds);
          float d0, d1;
          unpack_f32x2(mul_f32x2(p2[i], t), d0, d1);
          pk[i] = pack_bf16(d0, d1);
        }
        tmem_st_32x32(t_dp, pk);                    // over columns this warpgroup has consumed
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&ds_full[j & 1]);
    }
    if (nblk > 0) {
      if (!mbar_wait(&dq_full, 0)) { if (lane == 0) atomicExch(a.status, 59); goto teardown; }
      tc_fence_after();
    }
    __nv_bfloat16* drow = a.dq + (((size_t)b * a.S + (row_ok ? qi : 0)) * a.H + h) * D + wg * (D / 2);
#pragma unroll 1
    for (int c = 0; c < D / 2; c += 32) {
      uint32_t v[32];
      if (nblk > 0) {
        tmem_ld_32x32(tmem + lane_base + COL_DQ + wg * (D / 2) + c, v);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0u;
      }
      if (row_ok) {
#pragma unroll
        for (int i = 0; i < 32; i += 8)
          *reinterpret_cast<uint4*>(drow + c + i) =
              make_uint4(pack_bf16(__uint_as_float(v[i]), __uint_as_float(v[i + 1])),
                         pack_bf16(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])),
                         pack_bf16(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5])),
                         pack_bf16(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7])));
      }
    }
    tc_fence_before();
  }
teardown:
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

}  // namespace kmoe

// ------------------------------------------------------------------ host side
namespace kmoe {

// [B, S, Hx, D] bf16 tensor viewed as dims {D, Hx, S, B}; box = 64 columns of one head for `rows` positions.
static int make_bshd_tmap(CUtensorMap* out, const void* base, int B, int S, int Hx, int D, int rows) {
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)Hx, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 2, (cuuint64_t)Hx * D * 2, (cuuint64_t)S * Hx * D * 2};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)rows, 1};
  return encode_bf16_4d(out, base, dims, strides, box);
}

// Query tiles per CTA.  Two tiles keep the tensor pipe busier but slow each other down: a lone tile takes a key block in
// about 0.85 of a pair's time.  So one tile per CTA while all tiles run at once on the 148 SMs, and up to 4/3 of that where
// the causal mask makes enough of them short.  Forward us, two / one: 1x149x16 10.9 / 8.9, 1x777x12 20.2 / 17.6, 1x1536x12
// 32.4 / 27.7, 2x777x12 (1.1 waves) 21.7 / 18.5, 1x2048x12x64 (1.3) 34.5 / 29.0; beyond: 2x1002x16 (1.7) 24.9 / 26.5,
// 8x256x16 (1.7) 13.2 / 16.9, 4x1024x12 (2.6) 31.6 / 40.9.
template <int D>
static int launch_attn_fwd2(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, AttnArgs a,
                            cudaStream_t st) {
  const int smem = 6 * (D / 64) * PANEL_BYTES + 1024;
  auto kern = attn_fwd2_kernel<D>;
  static SmemLimit limit;
  if (!limit.raise(kern, smem)) return -20;
  const int blocks = (a.S + 127) / 128;
  const long long tiles = (long long)a.H * a.B * blocks;
  a.q_tiles = tiles <= 148 || (blocks >= 6 && 3 * tiles <= 4 * 148) ? 1 : 2;
  const int rows = 128 * a.q_tiles;
  dim3 grid(a.H, a.B, (a.S + rows - 1) / rows);
  kern<<<grid, F2_THREADS, smem, st>>>(tq, tk, tv, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // namespace kmoe

extern "C" int kmoe_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int H,
                             int Hkv, int D, float scale, const int* doc_start, int* status, cudaStream_t st) {
  using namespace kmoe;
  if (D != 64 && D != 128) return -1;
  if (H % Hkv) return -2;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_tmap(&tq, q, B, S, H, D, ATT_BLK))) return rc;
  if ((rc = make_bshd_tmap(&tk, k, B, S, Hkv, D, F2_KEYS))) return rc;
  if ((rc = make_bshd_tmap(&tv, v, B, S, Hkv, D, F2_KEYS))) return rc;
  AttnArgs a{B, S, H, Hkv, scale * 1.4426950408889634f, (__nv_bfloat16*)out, lse, status, doc_start, 2};
  return D == 128 ? launch_attn_fwd2<128>(tq, tk, tv, a, st) : launch_attn_fwd2<64>(tq, tk, tv, a, st);
}

namespace kmoe {

// CTAs that share a key block of the dK/dV kernel: 1, 2 or 4 out of the heads of the group.  Time is counted in steps:
// the first key block's CTA needs group * nb of them, divided by the split; an SM gets its share of all steps plus about
// eight for each CTA that it runs (prologue, epilogue, the sum over the cluster).  Measured us for 1 / 2 / 4 CTAs
// (head_dim 128 unless noted): 4x2048x16/4 123 / 154 / 224, 2x2048x16/4 114 / 78 / 115, 1x2048x16/4 110 / 64 / 58,
// 4x1024x12/3 64 / 45 / 66, 1x777x12/3 61 / 37 / 27, 8x1021x12/3x64 68 / 79 / 109, 1x64x8/2x64 16 / 14 / 12.
static int dkv_split(int nb, int Hkv, int B, int group, int sms) {
  const double ctas = (double)nb * Hkv * B / sms, steps = ctas * group * (nb + 1) / 2.0;
  int best = 1;
  double best_t = 1e30;
  for (int s = 1; s <= 4 && group % s == 0; s *= 2) {
    const double longest = (double)group * nb / s, share = steps + 8.0 * ctas * s;
    const double t = longest > share ? longest : share;
    if (t < best_t) { best_t = t; best = s; }
  }
  return best;
}

template <int D>
static int launch_attn_bwd(const void* q, const void* k, const void* v, const void* d_o, const AttnBwdArgs& a,
                           cudaStream_t st) {
  CUtensorMap tq, tdo, tk, tv;
  int rc;
  if ((rc = make_bshd_tmap(&tq, q, a.B, a.S, a.H, D, ATT_BLK))) return rc;
  if ((rc = make_bshd_tmap(&tdo, d_o, a.B, a.S, a.H, D, ATT_BLK))) return rc;
  if ((rc = make_bshd_tmap(&tk, k, a.B, a.S, a.Hkv, D, ATT_BLK))) return rc;
  if ((rc = make_bshd_tmap(&tv, v, a.B, a.S, a.Hkv, D, ATT_BLK))) return rc;
  constexpr int smem_dq = 7 * (D / 64) * PANEL_BYTES + 1024, smem_dkv = dkv2_smem_bytes<D>();
  static SmemLimit limit_dq, limit_dkv;
  if (!limit_dq.raise(attn_bwd_dq2_kernel<D>, smem_dq) || !limit_dkv.raise(attn_bwd_dkv2_kernel<D>, smem_dkv)) return -20;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    sms = n > 0 ? n : 148;
  }
  const int nb = (a.S + ATT_BLK - 1) / ATT_BLK;
  attn_bwd_dq2_kernel<D><<<dim3(a.H, a.B, nb), B2_THREADS, smem_dq, st>>>(tq, tdo, tk, tv, a);
  const int split = dkv_split(nb, a.Hkv, a.B, a.H / a.Hkv, sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.Hkv * split), (unsigned)a.B, (unsigned)nb);
  cfg.blockDim = dim3(B2_THREADS);
  cfg.dynamicSmemBytes = smem_dkv;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)split; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, attn_bwd_dkv2_kernel<D>, tq, tdo, tk, tv, a, split) != cudaSuccess) return -21;
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
}  // namespace kmoe

// stats is scratch of 2 * B * H * Sp floats, Sp = S rounded up to 128.
extern "C" int kmoe_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                             const float* lse, float* stats, void* dq, void* dk, void* dv, int B, int S, int H,
                             int Hkv, int D, float scale, const int* doc_start, int* status, cudaStream_t st) {
  using namespace kmoe;
  if (D != 64 && D != 128) return -1;
  if (H % Hkv) return -2;
  const int Sp = (S + ATT_BLK - 1) / ATT_BLK * ATT_BLK;
  const long long rows = (long long)B * Sp * H;
  if (rows == 0) return 0;
  float *nlse = stats, *ndelta = stats + rows;
  const int rows_per_block = 4 * 256 / (D / 8);
  const unsigned grid = (unsigned)((rows + rows_per_block - 1) / rows_per_block);
  if (D == 128)
    attn_stats_kernel<128><<<grid, 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, lse, nlse, ndelta,
                                                 rows, S, Sp, H, scale);
  else
    attn_stats_kernel<64><<<grid, 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, lse, nlse, ndelta,
                                                rows, S, Sp, H, scale);
  AttnBwdArgs a{B, S, H, Hkv, scale, scale * 1.4426950408889634f, Sp, nlse, ndelta, (__nv_bfloat16*)dq,
                (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, status, doc_start};
  return D == 128 ? launch_attn_bwd<128>(q, k, v, d_o, a, st) : launch_attn_bwd<64>(q, k, v, d_o, a, st);
}
