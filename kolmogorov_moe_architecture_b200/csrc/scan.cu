// Selective scan (Mamba), forward and backward, channels-last bf16 activations.
//
//   h_t[n] = exp(dt_t A[n]) h_{t-1}[n] + dt_t u_t B_t[n]        y_t = sum_n C_t[n] h_t[n] + D u_t   (* silu(z_t))
//
// Layout of the work: a CTA is two warps that share 16 channels and walk the sequence in chunks of 8 steps.  One carries
// the recurrence: a lane owns two neighbouring channels and four of their N = 16 states, as four packed fp32 pairs (a
// pair = one state of both channels; lane = channel pair + 8 * state group).  The other works a chunk ahead and a chunk
// behind: it copies the inputs (cp.async, 16-byte pieces), prepares what a step needs once per channel pair (softplus,
// gates, products; two (step, pair) items per lane, which keeps what finishing them takes), spreads B and C out as fp32,
// and when the lanes' sums over their states lie in shared memory adds the four state groups and finishes the steps.
// With 4 x 4096 channels this fills the chip with one pass over the sequence.  Fewer channels are cut into P segments
// that run in parallel (the recurrence is linear, so a segment started from zero only lacks
// decay(segment) * state_before):
//   forward : pass 1 computes each segment's end state from zero and its sum of dt; pass 2 starts every segment
//             from the true state (a short serial combination of the earlier segments) and writes y plus a
//             state checkpoint every 8 steps.
//   backward: pass 1 runs dL/dh backwards through each segment from zero; pass 2 starts from the true incoming
//             value, replays a chunk from its checkpoint and walks it in reverse, in halves of four steps whose decays and
//             states stay in registers; the later half comes first, so the earlier one is replayed twice.
// dB and dC are sums over channels: a lane adds its two channels, the warp lays four steps of its lanes' values out in
// shared memory and each lane of the other warp adds up eight 16-byte pieces and sends them off as one 16-byte global
// reduction.
//
// Bounds: the latency of a step with 1.7 recurrences per scheduler, beside the shared-memory pipe (44 and 62 % busy,
// forward and backward at 4 x 2048 x 4096) and the issue slots (54 and 50 %).  The exponentials alone take 119 us forward and
// 178 us backward (twelve steps' worth for eight).  Kernel times there: forward 341 -> 267 us, backward 832 -> 678;
// 1 x 2048 x 4096 in segments 137 + 270 -> 117 + 233; 1 x 333 x 1536 17 + 34 -> 15 + 30.  Against one channel per lane (the form before this) it is 0.65 of the instructions
// and half of the shared-memory reads per state.  Also measured: one warp doing everything 437 + 748 (too few warps to
// hide latency), eight recurrence warps of 200 registers beside eight of 56 in one CTA 970 backward (spills).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kmoe_api.h"
#include "ptx.cuh"

namespace kmoe {

constexpr int SN = 16;        // states
constexpr int CK = 8;         // checkpoint interval = steps per chunk
constexpr int WCH = 16;       // channels per warp
constexpr int NP = WCH / 2;   // channel pairs per warp
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

__device__ __forceinline__ void s_cp16(void* dst, const void* src, bool valid) {
  const uint32_t d = smem_u32(dst);
  const int sz = valid ? 16 : 0;   // src-size 0 zero-fills the destination
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}
__device__ __forceinline__ void s_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_>
__device__ __forceinline__ void s_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory"); }
__device__ __forceinline__ void s_red4(float* dst, float4 v) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
               ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ uint64_t s_dup(float v) { return pack_f32x2(v, v); }
__device__ __forceinline__ uint64_t s_ex2x2(uint64_t x) {
  float a, b;
  unpack_f32x2(x, a, b);
  return pack_f32x2(ex2_approx(a), ex2_approx(b));
}
__device__ __forceinline__ float s_hsum(uint64_t x) {
  float a, b;
  unpack_f32x2(x, a, b);
  return a + b;
}
__device__ __forceinline__ float s_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float s_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint64_t s_bf2(uint32_t w) { return pack_f32x2(s_lo(w), s_hi(w)); }
__device__ __forceinline__ uint32_t s_tobf2(uint64_t v) {
  float a, b;
  unpack_f32x2(v, a, b);
  return pack_bf16(a, b);
}
__device__ __forceinline__ uint64_t s_rcp2(uint64_t x) {
  float a, b;
  unpack_f32x2(x, a, b);
  return pack_f32x2(__fdividef(1.f, a), __fdividef(1.f, b));
}
// exp(-|x|), from which softplus and sigmoid of both signs follow without overflow
__device__ __forceinline__ uint64_t s_expnabs(uint64_t x) {
  float a, b;
  unpack_f32x2(x, a, b);
  return pack_f32x2(ex2_approx(-fabsf(a) * LOG2E), ex2_approx(-fabsf(b) * LOG2E));
}
// softplus(x) = max(x, 0) + log(1 + e), e = exp(-|x|): log(1 + e) = 2 atanh(r), r = e / (2 + e) <= 1/3, by its power
// series up to r^13 (the first term left out is 1.4e-8 of the sum)
__device__ __forceinline__ uint64_t s_softplus2(uint64_t x, uint64_t e) {
  const uint64_t r = mul_f32x2(e, s_rcp2(add_f32x2(e, s_dup(2.f))));
  const uint64_t q = mul_f32x2(r, r);
  uint64_t p = fma_f32x2(q, s_dup(2.f / 13.f), s_dup(2.f / 11.f));
  p = fma_f32x2(p, q, s_dup(2.f / 9.f));
  p = fma_f32x2(p, q, s_dup(2.f / 7.f));
  p = fma_f32x2(p, q, s_dup(2.f / 5.f));
  p = fma_f32x2(p, q, s_dup(2.f / 3.f));
  p = fma_f32x2(p, q, s_dup(2.f));
  float a, b;
  unpack_f32x2(x, a, b);
  // not fmaxf: a NaN has to come through
  return fma_f32x2(p, r, pack_f32x2(a < 0.f ? 0.f : a, b < 0.f ? 0.f : b));
}
// sigmoid(x) from e = exp(-|x|)
__device__ __forceinline__ uint64_t s_sigmoid2(uint64_t x, uint64_t e) {
  const uint64_t q = s_rcp2(add_f32x2(e, s_dup(1.f))), eq = mul_f32x2(e, q);
  float a, b, qa, qb, ea, eb;
  unpack_f32x2(x, a, b);
  unpack_f32x2(q, qa, qb);
  unpack_f32x2(eq, ea, eb);
  return pack_f32x2(a < 0.f ? ea : qa, b < 0.f ? eb : qb);
}

struct ScanArgs {
  const __nv_bfloat16* u;      // [B,S,C]
  const __nv_bfloat16* delta;  // [B,S,C]
  const __nv_bfloat16* z;      // [B,S,*] ld = ldz, may be null
  const float* A;              // [G,C,N]
  const void* Bm;              // [B,S,N], rows ldbc elements apart, bf16 or fp32
  const void* Cm;
  const float* D;              // [G,C] or null
  const float* dt_bias;        // [G,C] or null
  int S, C;
  long long ldz, ldbc;
  int softplus;
  int bpg;                     // batch entries per parameter set
  int P, seg_len;              // segments, steps per segment (multiple of CK)
};

// seg scratch: [B, P, C, SN] end states of the segments started from zero, then [B, P, C] sums of dt
__device__ __forceinline__ size_t seg_row(const ScanArgs& a, int b, int p, int c) { return ((size_t)b * a.P + p) * a.C + c; }

// Inputs of one chunk.  T: element type of B and C.
template <typename T>
struct __align__(16) RawTile {
  __nv_bfloat16 x[4][CK][WCH];                 // which four arrays is the kernel's business
  T bc[2][CK][SN];
};
// Staging of a chunk: a row of an array is two 16-byte pieces; a lane copies one piece of one step of arrays lane / 16
// and 2 + lane / 16, and one or two pieces of B and C.  Nothing but the sources (kernel arguments, null = nothing to copy)
// outlives a call: the registers are wanted elsewhere.
struct Sources {
  const __nv_bfloat16* s[4];
  long long ld[4];
};
template <typename T, bool WANT_B, bool WANT_C>
__device__ __forceinline__ void load_tile(RawTile<T>& st, const ScanArgs& a, const Sources& src, int b, int cw, int t0,
                                          int t_end, int lane) {
  constexpr int PIECES = SN * (int)sizeof(T) / 16, PER_LANE = 2 * CK * PIECES / 32;      // pieces of a row of B or C
  const int row = (lane >> 1) & 7, t = t0 + row, ch = (lane & 1) * 8;
  const bool have = cw + ch < a.C;
  const size_t rowid = (size_t)b * a.S + (t < t_end ? t : t_end - 1);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const __nv_bfloat16* p = lane < 16 ? src.s[2 * k] : src.s[2 * k + 1];
    const long long ld = lane < 16 ? src.ld[2 * k] : src.ld[2 * k + 1];
    if (p != nullptr)
      s_cp16(&st.x[2 * k + (lane >> 4)][row][ch], p + rowid * ld + cw + (have ? ch : 0), have && t < t_end);
  }
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int j = lane + 32 * i, which = j / (CK * PIECES), r2 = (j / PIECES) % CK, pt = j % PIECES, t2 = t0 + r2;
    if (which ? WANT_C : WANT_B)
      s_cp16(&st.bc[which][r2][pt * (16 / (int)sizeof(T))],
             reinterpret_cast<const T*>(which ? a.Cm : a.Bm) + ((size_t)b * a.S + (t2 < t_end ? t2 : t_end - 1)) * a.ldbc +
                 pt * (16 / (int)sizeof(T)),
             t2 < t_end);
  }
  s_commit();
}

// B and C of a chunk as fp32.  A packed operation takes one value for both halves of an operand at no cost, so they are
// not written twice.
struct __align__(16) BC32 {
  float v[2][CK][SN];
};
__device__ __forceinline__ void bc_fill(BC32& d, const __nv_bfloat16 (&bc)[2][CK][SN], int lane) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint2 q = reinterpret_cast<const uint2*>(&bc)[lane + 32 * j];
    reinterpret_cast<float4*>(&d)[lane + 32 * j] = make_float4(s_lo(q.x), s_hi(q.x), s_lo(q.y), s_hi(q.y));
  }
}
__device__ __forceinline__ void bc_fill(BC32& d, const float (&bc)[2][CK][SN], int lane) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
    reinterpret_cast<float4*>(&d)[lane + 32 * j] = reinterpret_cast<const float4*>(&bc)[lane + 32 * j];
}
// the four states of group sg of one step, each for both channels
__device__ __forceinline__ void bc_load(const BC32& d, int which, int step, int sg, uint64_t (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(&d.v[which][step][sg * 4]);
  v[0] = s_dup(q.x);
  v[1] = s_dup(q.y);
  v[2] = s_dup(q.z);
  v[3] = s_dup(q.w);
}
// rows of two channels <-> packed pairs
__device__ __forceinline__ void pair_rows(float4 x, float4 y, uint64_t (&v)[4]) {
  v[0] = pack_f32x2(x.x, y.x);
  v[1] = pack_f32x2(x.y, y.y);
  v[2] = pack_f32x2(x.z, y.z);
  v[3] = pack_f32x2(x.w, y.w);
}
__device__ __forceinline__ void unpair_rows(const uint64_t (&v)[4], float4& x, float4& y) {
  unpack_f32x2(v[0], x.x, y.x);
  unpack_f32x2(v[1], x.y, y.y);
  unpack_f32x2(v[2], x.z, y.z);
  unpack_f32x2(v[3], x.w, y.w);
}
// Fetches four states of channels c and c + 1 from rows of SN floats; a pair past the last channel reads as zero.
__device__ __forceinline__ void load_rows(const float* p, bool ok, float4& x, float4& y) {
  x = ok ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
  y = ok ? __ldg(reinterpret_cast<const float4*>(p + SN)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void store_rows(float* p, const uint64_t (&v)[4]) {
  float4 x, y;
  unpair_rows(v, x, y);
  *reinterpret_cast<float4*>(p) = x;
  *reinterpret_cast<float4*>(p + SN) = y;
}
// A checkpoint keeps the 16 channels of a warp as its lanes hold them: 2 x 32 pieces of 16 bytes, [pair of states][lane].
__device__ __forceinline__ size_t ckpt_row(const ScanArgs& a, int b, int chunk, int block) {
  return (((size_t)b * ((a.S + CK - 1) / CK) + chunk) * ((a.C + WCH - 1) / WCH) + block) * (WCH * SN);
}
__device__ __forceinline__ void load_decay(const ScanArgs& a, int pc, int sg, bool ok, uint64_t (&An)[4]) {
  float4 x, y;
  load_rows(a.A + (size_t)pc * SN + sg * 4, ok, x, y);
  pair_rows(x, y, An);
#pragma unroll
  for (int k = 0; k < 4; ++k) An[k] = mul_f32x2(An[k], s_dup(LOG2E));
}
__device__ __forceinline__ uint64_t load_pair(const float* p, int pc, bool ok) {
  return p != nullptr && ok ? pack_f32x2(p[pc], p[pc + 1]) : 0ull;
}
// x[pair sums of four steps][lane] -> sum over the state groups of one step's pair; the lanes of a step start at
// different groups, which keeps their reads on different banks
__device__ __forceinline__ uint64_t sum_groups(const float2 (&x)[32], int step, int cp) {
  uint64_t s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t q = *reinterpret_cast<const uint64_t*>(&x[((k + step) & 3) * 8 + cp]);
    s = k == 0 ? q : add_f32x2(s, q);
  }
  return s;
}

// Which of a CTA's two warps carries the recurrence.  A warp's scheduler follows from its slot on the SM, and CTAs of two
// warps take slots in twos: with the same role for the same warp of every CTA, the recurrences would share two of the
// SM's four schedulers.  So the roles are swapped in every second pair of slots (the slot number is a hint: the choice
// is made once per CTA and only speed depends on it).
__device__ __forceinline__ bool is_helper(uint32_t* shared_flip) {
  if (threadIdx.x == 0) {
    uint32_t slot;
    asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
    *shared_flip = (slot >> 2) & 1;
  }
  __syncthreads();
  return ((threadIdx.x >> 5) ^ *shared_flip) != 0;
}
// Forward: the two warps meet after every chunk (handing over as below, with the finishing a chunk later, was 4 % slower).
__device__ __forceinline__ void pair_step() { asm volatile("bar.sync 1, 64;" ::: "memory"); }
// Backward: the one that goes on arrives, the one that needs the data (or the buffer) syncs.
// READY + parity: a chunk is prepared.  FULL + i: results of buffer i are written.  EMPTY + i: they have been read.
enum : int { READY = 1, FULL = 3, EMPTY = 5 };
template <int ID>
__device__ __forceinline__ void pair_arrive(int which) {
  if (which) asm volatile("bar.arrive %0, 64;" ::"n"(ID + 1) : "memory");
  else asm volatile("bar.arrive %0, 64;" ::"n"(ID) : "memory");
}
template <int ID>
__device__ __forceinline__ void pair_sync(int which) {
  if (which) asm volatile("bar.sync %0, 64;" ::"n"(ID + 1) : "memory");
  else asm volatile("bar.sync %0, 64;" ::"n"(ID) : "memory");
}

// MODE 0: end state from zero + sum of dt (segments 0 .. P-2).  MODE 1: outputs and checkpoints.
template <int MODE, typename T>
__global__ void __launch_bounds__(64)
scan_fwd_kernel(ScanArgs a, __nv_bfloat16* __restrict__ out, float* __restrict__ ckpt, float* __restrict__ seg) {
  struct __align__(16) Shared {
    RawTile<T> st[2];
    BC32 bc[2];
    float4 sc[2][CK][NP];                      // dt, dt * u of a pair
    float2 part[2][CK][32];                    // every lane's sums over its states
    uint32_t y[CK][NP];
  };
  __shared__ Shared w;
  __shared__ uint32_t flip;
  const int lane = threadIdx.x & 31, cp = lane & 7, sg = lane >> 3;
  const int cw = blockIdx.x * WCH, c = cw + 2 * cp, p = blockIdx.y, b = blockIdx.z;
  const bool live = c < a.C;                   // C is a multiple of 8: a pair exists or does not, as a whole
  const int pc = (b / a.bpg) * a.C + c;
  const int t_begin = p * a.seg_len, t_end = min(a.S, t_begin + a.seg_len);
  const int ntiles = (t_end - t_begin + CK - 1) / CK;
  const size_t nrows = (size_t)gridDim.z * a.P * a.C;      // rows of the segment scratch

  if (is_helper(&flip)) {                      // ---- the warp that prepares and finishes chunks
    const bool has_z = a.z != nullptr;
    const uint64_t Dc = load_pair(a.D, pc, live), bias = load_pair(a.dt_bias, pc, live);
    const Sources src = {{a.u, a.delta, MODE == 1 ? a.z : nullptr, nullptr}, {a.C, a.C, a.ldz, 0}};
    auto stage = [&](int tile) {
      if (tile < ntiles) load_tile<T, true, MODE == 1>(w.st[tile & 1], a, src, b, cw, t_begin + tile * CK, t_end, lane);
      else s_commit();
    };
    struct Item {                              // what finishing step sg (+ 4) of this lane's channels takes
      uint64_t du, gate;
    };
    struct Items {
      Item k[2];
    } cur, nxt;
    auto prepare = [&](int tile, Items& it) {
      const RawTile<T>& st = w.st[tile & 1];
      const int t0 = t_begin + tile * CK, par = tile & 1;
      bc_fill(w.bc[par], st.bc, lane);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = sg + 4 * k;
        const bool ok = t0 + row < t_end;      // steps past the end leave the state alone
        const uint64_t uu = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[0][row][2 * cp]));
        uint64_t dt = add_f32x2(s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[1][row][2 * cp])), bias);
        if (a.softplus) dt = s_softplus2(dt, s_expnabs(dt));
        if (!ok) dt = 0;
        *reinterpret_cast<ulonglong2*>(&w.sc[par][row][cp]) = make_ulonglong2(dt, ok ? mul_f32x2(dt, uu) : 0ull);
        if (MODE == 1) {
          it.k[k].du = mul_f32x2(Dc, uu);
          it.k[k].gate = s_dup(1.f);
          if (has_z) {
            const uint64_t zv = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[2][row][2 * cp]));
            it.k[k].gate = mul_f32x2(zv, s_sigmoid2(zv, s_expnabs(zv)));
          }
        }
      }
    };
    auto finish = [&](int tile, const Items& it) {
      const int t0 = t_begin + tile * CK, par = tile & 1;
#pragma unroll
      for (int k = 0; k < 2; ++k)
        w.y[sg + 4 * k][cp] =
            s_tobf2(mul_f32x2(add_f32x2(sum_groups(w.part[par][sg + 4 * k], sg, cp), it.k[k].du), it.k[k].gate));
      __syncwarp();
      const int row = lane >> 1, ch = (lane & 1) * 8;
      if (lane < 2 * CK && t0 + row < t_end && cw + ch < a.C)
        *reinterpret_cast<uint4*>(out + ((size_t)b * a.S + t0 + row) * a.C + cw + ch) =
            *reinterpret_cast<const uint4*>(&w.y[row][ch / 2]);
    };
    stage(0);
    stage(1);
    s_wait<1>();
    __syncwarp();
    prepare(0, nxt);
    pair_step();
    for (int tile = 0; tile < ntiles; ++tile) {          // the other warp is at chunk `tile`
      if (MODE == 1 && tile > 0) finish(tile - 1, cur);
      cur = nxt;
      stage(tile + 2);
      s_wait<1>();
      __syncwarp();
      if (tile + 1 < ntiles) prepare(tile + 1, nxt);
      pair_step();
    }
    if (MODE == 1) finish(ntiles - 1, cur);
    return;
  }

  // ---- the warp that carries the recurrence
  uint64_t An[4], h[4] = {0, 0, 0, 0};
  load_decay(a, pc, sg, live, An);
  if (MODE == 1 && live) {
    // state before this segment: fold the earlier segments' zero-started end states, oldest first
    for (int q = 0; q < p; ++q) {
      const size_t r = seg_row(a, b, q, c);
      const uint64_t sdt = pack_f32x2(seg[nrows * SN + r], seg[nrows * SN + r + 1]);
      uint64_t e[4];
      pair_rows(*reinterpret_cast<const float4*>(seg + r * SN + sg * 4),
                *reinterpret_cast<const float4*>(seg + (r + 1) * SN + sg * 4), e);
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = fma_f32x2(s_ex2x2(mul_f32x2(An[k], sdt)), h[k], e[k]);
    }
  }
  uint64_t sdt = 0;
  float* ck = MODE == 1 && ckpt != nullptr ? ckpt + ckpt_row(a, b, t_begin / CK, blockIdx.x) + lane * 4 : nullptr;
  const size_t ck_step = (size_t)gridDim.x * (WCH * SN);
  pair_step();
  for (int tile = 0; tile < ntiles; ++tile) {
    const int par = tile & 1;
    if (MODE == 1 && ck != nullptr) {
      *reinterpret_cast<ulonglong2*>(ck) = make_ulonglong2(h[0], h[1]);
      *reinterpret_cast<ulonglong2*>(ck + 128) = make_ulonglong2(h[2], h[3]);
      ck += ck_step;
    }
    // no store to shared memory before the chunk's last read: it would keep the reads of later steps behind it
    uint64_t ys[CK];
#pragma unroll
    for (int i = 0; i < CK; ++i) {
      const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(&w.sc[par][i][cp]);
      uint64_t Bv[4];
      bc_load(w.bc[par], 0, i, sg, Bv);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        h[k] = fma_f32x2(s_ex2x2(mul_f32x2(d.x, An[k])), h[k], mul_f32x2(d.y, Bv[k]));
      if (MODE == 1) {
        uint64_t Cv[4];
        bc_load(w.bc[par], 1, i, sg, Cv);
        ys[i] = mul_f32x2(Cv[0], h[0]);
#pragma unroll
        for (int k = 1; k < 4; ++k) ys[i] = fma_f32x2(Cv[k], h[k], ys[i]);
      } else {
        sdt = add_f32x2(sdt, d.x);
      }
    }
    if (MODE == 1) {
#pragma unroll
      for (int i = 0; i < CK; ++i) *reinterpret_cast<uint64_t*>(&w.part[par][i][lane]) = ys[i];
    }
    pair_step();
  }
  if (MODE == 0 && live) {
    const size_t r = seg_row(a, b, p, c);
    store_rows(seg + r * SN + sg * 4, h);
    if (sg == 0) unpack_f32x2(sdt, seg[nrows * SN + r], seg[nrows * SN + r + 1]);
  }
}

// ------------------------------------------------------------------ backward, pass 1
// dL/dh carried backwards through segment p (1 .. P-1) from zero: gseg[b][p][c][n] = what the segment hands to
// the step before its first one.
template <typename T>
__global__ void __launch_bounds__(64)
scan_bwd_carry_kernel(ScanArgs a, const __nv_bfloat16* __restrict__ dout, float* __restrict__ gseg) {
  struct __align__(16) Shared {
    RawTile<T> st[2];
    BC32 bc[2];
    float4 sc[2][CK][NP];                      // dt, dL/dy of a pair
  };
  __shared__ Shared w;
  __shared__ uint32_t flip;
  const int lane = threadIdx.x & 31, cp = lane & 7, sg = lane >> 3;
  const int cw = blockIdx.x * WCH, c = cw + 2 * cp, p = blockIdx.y + 1, b = blockIdx.z;
  const bool live = c < a.C;
  const int pc = (b / a.bpg) * a.C + c;
  const int t_begin = p * a.seg_len, t_end = min(a.S, t_begin + a.seg_len);
  const int ntiles = (t_end - t_begin + CK - 1) / CK;

  if (is_helper(&flip)) {
    const bool has_z = a.z != nullptr;
    const uint64_t bias = load_pair(a.dt_bias, pc, live);
    const Sources src = {{a.delta, a.z, dout, nullptr}, {a.C, a.ldz, a.C, 0}};
    auto stage = [&](int j) {                  // j-th chunk from the end
      if (j < ntiles) load_tile<T, false, true>(w.st[j & 1], a, src, b, cw, t_begin + (ntiles - 1 - j) * CK, t_end, lane);
      else s_commit();
    };
    auto prepare = [&](int j) {
      const RawTile<T>& st = w.st[j & 1];
      const int t0 = t_begin + (ntiles - 1 - j) * CK, par = j & 1;
      bc_fill(w.bc[par], st.bc, lane);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = sg + 4 * k;
        uint64_t dt = add_f32x2(s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[0][row][2 * cp])), bias);
        if (a.softplus) dt = s_softplus2(dt, s_expnabs(dt));
        uint64_t dy = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[2][row][2 * cp]));
        if (has_z) {
          const uint64_t zv = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[1][row][2 * cp]));
          dy = mul_f32x2(dy, mul_f32x2(zv, s_sigmoid2(zv, s_expnabs(zv))));
        }
        *reinterpret_cast<ulonglong2*>(&w.sc[par][row][cp]) =
            t0 + row < t_end ? make_ulonglong2(dt, dy) : make_ulonglong2(0, 0);
      }
    };
    stage(0);
    stage(1);
    s_wait<1>();
    __syncwarp();
    prepare(0);
    pair_arrive<READY>(0);
    for (int j = 0; j + 1 < ntiles; ++j) {
      stage(j + 2);
      s_wait<1>();
      __syncwarp();
      if (j > 0) pair_sync<EMPTY>((j + 1) & 1);
      prepare(j + 1);
      pair_arrive<READY>((j + 1) & 1);
    }
    return;
  }
  uint64_t An[4], g[4] = {0, 0, 0, 0};
  load_decay(a, pc, sg, live, An);
  for (int j = 0; j < ntiles; ++j) {
    const int par = j & 1;
    pair_sync<READY>(par);
#pragma unroll
    for (int i = CK - 1; i >= 0; --i) {
      const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(&w.sc[par][i][cp]);
      uint64_t Cv[4];
      bc_load(w.bc[par], 1, i, sg, Cv);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        g[k] = mul_f32x2(fma_f32x2(Cv[k], d.y, g[k]), s_ex2x2(mul_f32x2(d.x, An[k])));
    }
    if (j + 2 < ntiles) pair_arrive<EMPTY>(par);
  }
  if (live) store_rows(gseg + seg_row(a, b, p, c) * SN + sg * 4, g);
}

// ------------------------------------------------------------------ backward, pass 2
// A chunk is replayed in halves of four steps, the earlier one twice: decays and states of eight steps would be 128
// registers, and with those only four such pairs of warps would fit on an SM.
template <typename T>
struct __align__(16) BwdShared {               // of one pair of warps
  RawTile<T> st[2];                            // u, delta, z, dout
  ulonglong2 ck[3][2][32];                     // the states before the chunk, as the lanes hold them
  BC32 bc[2];
  float4 s1[2][CK][NP];                        // dt, dt * u of a pair of channels
  float2 s2[2][CK][NP];                        // dL/dy
  uint32_t o[3][CK][NP];                       // du, ddelta, dz
  float2 sums[2][3][4][32];                    // by half: four steps of every lane's three sums over its states
  float4 part[2][4][2][32];                    // by half: four steps of every lane's dB and dC
};

template <typename T>
__global__ void __launch_bounds__(64, 7)
scan_bwd_kernel(ScanArgs a, const __nv_bfloat16* __restrict__ dout, const float* __restrict__ ckpt,
                const float* __restrict__ seg, const float* __restrict__ gseg, __nv_bfloat16* __restrict__ du,
                __nv_bfloat16* __restrict__ ddelta, __nv_bfloat16* __restrict__ dz, long long lddz,
                float* __restrict__ dA, float* __restrict__ dB, float* __restrict__ dC, float* __restrict__ dD,
                float* __restrict__ dbias) {
  __shared__ BwdShared<T> w;
  __shared__ uint32_t flip;
  const int lane = threadIdx.x & 31, cp = lane & 7, sg = lane >> 3;
  const int cw = blockIdx.x * WCH, c = cw + 2 * cp, p = blockIdx.y, b = blockIdx.z;
  const bool live = c < a.C;                   // a pair past the last channel computes on zeros and stores nothing
  const int pc = (b / a.bpg) * a.C + c;
  const int t_begin = p * a.seg_len, t_end = min(a.S, t_begin + a.seg_len);
  const int ntiles = (t_end - t_begin + CK - 1) / CK;

  if (is_helper(&flip)) {
    const bool has_z = a.z != nullptr;
    const uint64_t Dc = load_pair(a.D, pc, live), bias = load_pair(a.dt_bias, pc, live);
    uint64_t dDacc = 0, dbacc = 0;
    const Sources src = {{a.u, a.delta, a.z, dout}, {a.C, a.C, a.ldz, a.C}};
    auto stage = [&](int j) {                  // j-th chunk from the end
      if (j < ntiles) {
        const float* rows = ckpt + ckpt_row(a, b, t_begin / CK + ntiles - 1 - j, blockIdx.x);
#pragma unroll
        for (int k = 0; k < 2; ++k) s_cp16(&w.ck[j % 3][k][lane], rows + (k * 32 + lane) * 4, true);
        load_tile<T, true, true>(w.st[j & 1], a, src, b, cw, t_begin + (ntiles - 1 - j) * CK, t_end, lane);
      } else {
        s_commit();
      }
    };
    struct Item {                              // what finishing step sg (+ 4) of this lane's channels takes
      uint64_t dt, u, dy, zf, slope;           // zf: dz / y, slope: softplus'
    };
    struct Items {
      Item k[2];
    } cur, nxt;
    auto prepare = [&](int j, Items& it) {
      const RawTile<T>& st = w.st[j & 1];
      const int t0 = t_begin + (ntiles - 1 - j) * CK, par = j & 1;
      bc_fill(w.bc[par], st.bc, lane);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = sg + 4 * k;
        const bool ok = live && t0 + row < t_end;          // steps past the end: decay 1, nothing added, nothing summed
        const uint64_t uu = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[0][row][2 * cp]));
        uint64_t dt = add_f32x2(s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[1][row][2 * cp])), bias);
        uint64_t slope = s_dup(1.f);
        if (a.softplus) {
          const uint64_t e = s_expnabs(dt);
          slope = s_sigmoid2(dt, e);
          dt = s_softplus2(dt, e);
        }
        uint64_t dy = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[3][row][2 * cp])), zf = 0;
        if (has_z) {
          const uint64_t zv = s_bf2(*reinterpret_cast<const uint32_t*>(&st.x[2][row][2 * cp]));
          const uint64_t sgm = s_sigmoid2(zv, s_expnabs(zv));
          // silu'(z) = sgm (1 + z (1 - sgm))
          const uint64_t rest = fma_f32x2(sgm, s_dup(-1.f), s_dup(1.f));
          zf = mul_f32x2(mul_f32x2(dy, sgm), fma_f32x2(zv, rest, s_dup(1.f)));
          dy = mul_f32x2(dy, mul_f32x2(zv, sgm));
        }
        it.k[k] = ok ? Item{dt, uu, dy, zf, slope} : Item{0, 0, 0, 0, 0};
        *reinterpret_cast<ulonglong2*>(&w.s1[par][row][cp]) = make_ulonglong2(it.k[k].dt, mul_f32x2(it.k[k].dt, it.k[k].u));
        *reinterpret_cast<uint64_t*>(&w.s2[par][row][cp]) = it.k[k].dy;
      }
    };
    auto finish = [&](int j, int half, const Item& it) {   // this lane finishes step half * 4 + sg of its pair
      const int i = half * 4 + sg, t0 = t_begin + (ntiles - 1 - j) * CK;
      const uint64_t tA = sum_groups(w.sums[half][0][sg], sg, cp), tB = sum_groups(w.sums[half][1][sg], sg, cp),
                     tY = sum_groups(w.sums[half][2][sg], sg, cp);
      const uint64_t dd = mul_f32x2(fma_f32x2(tA, s_dup(LN2), mul_f32x2(it.u, tB)), it.slope);
      dDacc = fma_f32x2(it.dy, it.u, dDacc);
      dbacc = add_f32x2(dbacc, dd);
      w.o[0][i][cp] = s_tobf2(fma_f32x2(it.dt, tB, mul_f32x2(it.dy, Dc)));
      w.o[1][i][cp] = s_tobf2(dd);
      w.o[2][i][cp] = s_tobf2(mul_f32x2(it.zf, fma_f32x2(Dc, it.u, tY)));
      // channel sums: this lane takes four values (dB or dC of state group lane & 3) of step lane / 8; the lanes of a
      // step start at different channels, which keeps their 16-byte reads on different banks
      uint64_t acc[2] = {0, 0};
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(
            &w.part[half][sg][(lane >> 2) & 1][(lane & 3) * 8 + ((k + lane) & 7)]);
        acc[0] = k == 0 ? x.x : add_f32x2(acc[0], x.x);
        acc[1] = k == 0 ? x.y : add_f32x2(acc[1], x.y);
      }
      float4 v;
      unpack_f32x2(acc[0], v.x, v.y);
      unpack_f32x2(acc[1], v.z, v.w);
      const int t = t0 + i;
      if (t < t_end) s_red4(((lane & 4) ? dC : dB) + ((size_t)b * a.S + t) * SN + (lane & 3) * 4, v);
    };
    auto store = [&](int j) {
      const int t0 = t_begin + (ntiles - 1 - j) * CK;
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 2; ++k) {            // rows of du and ddelta, then of dz
        const int i = lane + 32 * k, arr = i >> 4, row = (i >> 1) & 7, ch = (i & 1) * 8, t = t0 + row;
        if (arr < (has_z ? 3 : 2) && t < t_end && cw + ch < a.C) {
          __nv_bfloat16* dst = arr == 0 ? du : (arr == 1 ? ddelta : dz);
          *reinterpret_cast<uint4*>(dst + ((size_t)b * a.S + t) * (arr == 2 ? lddz : (long long)a.C) + cw + ch) =
              *reinterpret_cast<const uint4*>(&w.o[arr][row][ch / 2]);
        }
      }
      __syncwarp();
    };
    stage(0);
    stage(1);
    s_wait<1>();
    __syncwarp();
    prepare(0, nxt);
    pair_arrive<READY>(0);
    for (int j = 0; j < ntiles; ++j) {
      if (j > 0) {                             // the other warp is in the later half of chunk j
        pair_sync<FULL>(0);
        finish(j - 1, 0, cur.k[0]);
        pair_arrive<EMPTY>(0);
        store(j - 1);
      }
      cur = nxt;
      stage(j + 2);
      s_wait<1>();
      __syncwarp();
      if (j + 1 < ntiles) {
        prepare(j + 1, nxt);
        pair_arrive<READY>((j + 1) & 1);
      }
      pair_sync<FULL>(1);                     // and now in its earlier half
      finish(j, 1, cur.k[1]);
      if (j + 1 < ntiles) pair_arrive<EMPTY>(1);
    }
    pair_sync<FULL>(0);
    finish(ntiles - 1, 0, cur.k[0]);
    store(ntiles - 1);
    float d0, d1, b0, b1;
    unpack_f32x2(dDacc, d0, d1);
    unpack_f32x2(dbacc, b0, b1);
#pragma unroll
    for (int k = 8; k <= 16; k <<= 1) {
      d0 += __shfl_xor_sync(0xffffffffu, d0, k);
      d1 += __shfl_xor_sync(0xffffffffu, d1, k);
      b0 += __shfl_xor_sync(0xffffffffu, b0, k);
      b1 += __shfl_xor_sync(0xffffffffu, b1, k);
    }
    if (live && sg == 0 && dD) {
      atomicAdd(&dD[pc], d0);
      atomicAdd(&dD[pc + 1], d1);
    }
    if (live && sg == 0 && dbias) {
      atomicAdd(&dbias[pc], b0);
      atomicAdd(&dbias[pc + 1], b1);
    }
    return;
  }

  uint64_t An[4], g[4] = {0, 0, 0, 0}, dAacc[4] = {0, 0, 0, 0};
  load_decay(a, pc, sg, live, An);
  // dL/dh flowing into the last step of this segment: fold the later segments' zero-started carries, last first
  if (live) {
    const size_t nrows = (size_t)gridDim.z * a.P * a.C;
    for (int q = a.P - 1; q > p; --q) {
      const size_t r = seg_row(a, b, q, c);
      const uint64_t sdt = q < a.P - 1 ? pack_f32x2(seg[nrows * SN + r], seg[nrows * SN + r + 1]) : 0ull;
      uint64_t e[4];
      pair_rows(*reinterpret_cast<const float4*>(gseg + r * SN + sg * 4),
                *reinterpret_cast<const float4*>(gseg + (r + 1) * SN + sg * 4), e);
#pragma unroll
      for (int k = 0; k < 4; ++k) g[k] = fma_f32x2(s_ex2x2(mul_f32x2(An[k], sdt)), g[k], e[k]);
    }
  }
  for (int j = 0, third = 0; j < ntiles; ++j, third = third == 2 ? 0 : third + 1) {
    const int par = j & 1;
    pair_sync<READY>(par);
    auto first_state = [&](uint64_t (&v)[4]) {
      const ulonglong2 x = w.ck[third][0][lane], y = w.ck[third][1][lane];
      v[0] = x.x;
      v[1] = x.y;
      v[2] = y.x;
      v[3] = y.y;
    };
    uint64_t hs[4];                            // state before the half at hand
    first_state(hs);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(&w.s1[par][i][cp]);
      uint64_t Bv[4];
      bc_load(w.bc[par], 0, i, sg, Bv);
#pragma unroll
      for (int k = 0; k < 4; ++k) hs[k] = fma_f32x2(s_ex2x2(mul_f32x2(d.x, An[k])), hs[k], mul_f32x2(d.y, Bv[k]));
    }
#pragma unroll
    for (int half = 1; half >= 0; --half) {
      // replay the half forward: decay of every step and state after it
      if (half == 0) first_state(hs);
      uint64_t an[4][4], h[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(&w.s1[par][half * 4 + i][cp]);
        uint64_t Bv[4];
        bc_load(w.bc[par], 0, half * 4 + i, sg, Bv);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          an[i][k] = s_ex2x2(mul_f32x2(d.x, An[k]));
          h[i][k] = fma_f32x2(an[i][k], i > 0 ? h[i - 1][k] : hs[k], mul_f32x2(d.y, Bv[k]));
        }
      }
      // reverse sweep
      if (j > 0) pair_sync<EMPTY>(half);
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(&w.s1[par][half * 4 + i][cp]);
        const uint64_t dy = *reinterpret_cast<const uint64_t*>(&w.s2[par][half * 4 + i][cp]);
        uint64_t Bv[4], Cv[4], sA, sB, sY;
        bc_load(w.bc[par], 0, half * 4 + i, sg, Bv);
        bc_load(w.bc[par], 1, half * 4 + i, sg, Cv);
        float vB[4], vC[4];                    // dB and dC of the lane's four states, both channels
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sY = k == 0 ? mul_f32x2(Cv[k], h[i][k]) : fma_f32x2(Cv[k], h[i][k], sY);
          vC[k] = s_hsum(mul_f32x2(dy, h[i][k]));
          const uint64_t gn = fma_f32x2(Cv[k], dy, g[k]);                // dL/dh_t
          sB = k == 0 ? mul_f32x2(gn, Bv[k]) : fma_f32x2(gn, Bv[k], sB);
          vB[k] = s_hsum(mul_f32x2(gn, d.y));
          g[k] = mul_f32x2(gn, an[i][k]);                                // handed to step t - 1
          const uint64_t gh = mul_f32x2(g[k], i > 0 ? h[i - 1][k] : hs[k]);
          sA = k == 0 ? mul_f32x2(gh, An[k]) : fma_f32x2(gh, An[k], sA);
          dAacc[k] = fma_f32x2(gh, d.x, dAacc[k]);
        }
        w.part[half][i][0][lane] = make_float4(vB[0], vB[1], vB[2], vB[3]);
        w.part[half][i][1][lane] = make_float4(vC[0], vC[1], vC[2], vC[3]);
        *reinterpret_cast<uint64_t*>(&w.sums[half][0][i][lane]) = sA;
        *reinterpret_cast<uint64_t*>(&w.sums[half][1][i][lane]) = sB;
        *reinterpret_cast<uint64_t*>(&w.sums[half][2][i][lane]) = sY;
      }
      pair_arrive<FULL>(half);
    }
  }
  if (live) {
    float4 x, y;
    unpair_rows(dAacc, x, y);
    s_red4(dA + (size_t)pc * SN + sg * 4, x);
    s_red4(dA + (size_t)(pc + 1) * SN + sg * 4, y);
  }
}

// Segment count: the one that minimises (rounds of CTAs per SM) x (steps per segment).  Up to about four CTAs on an
// SM the time of a step is its latency, beyond that it grows with the CTAs; cutting the sequence at all costs a second
// pass over it (about half of the work again).  Forward + backward of 1 x 2048 x 4096: 670 us in one segment and 382 in
// four when a lane had one channel, 371 in four now.
// Segments are multiples of the chunk and at least 64 steps long.
static void plan(int B, int S, int C, int* P, int* seg_len) {
  const long long per_seg = (long long)((C + WCH - 1) / WCH) * B;
  const long long sms = 148;
  double best_cost = -1;
  int best_len = (S + CK - 1) / CK * CK;
  for (int want = 1; want <= 32; ++want) {
    int len = (S + want - 1) / want;
    if (len < 64) len = 64;
    len = (len + CK - 1) / CK * CK;
    const int p = (S + len - 1) / len;
    const long long rounds = (per_seg * p + sms - 1) / sms;
    const double cost = (rounds < 4 ? 4.0 : (double)rounds) * len * (p > 1 ? 1.5 : 1.0);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best_len = len;
    }
  }
  if (best_len < CK) best_len = CK;
  *seg_len = best_len;
  *P = (S + best_len - 1) / best_len;
  if (*P < 1) *P = 1;
}

static int check(const ScanArgs& a, int bc_bf16, int B, int N, int groups) {
  if (N != SN || groups < 1 || B % groups) return -1;
  if (a.C % 8 || (a.z != nullptr && a.ldz % 8)) return -4;
  // rows of B and C are copied in 16-byte pieces
  if (a.ldbc % (bc_bf16 ? 8 : 4) || (reinterpret_cast<uintptr_t>(a.Bm) | reinterpret_cast<uintptr_t>(a.Cm)) & 15) return -6;
  return 0;
}

template <typename T>
static int launch_fwd(const ScanArgs& a, void* out, float* ckpt, float* seg, int B, cudaStream_t st) {
  const int nx = (a.C + WCH - 1) / WCH;
  if (a.P > 1) scan_fwd_kernel<0, T><<<dim3(nx, a.P - 1, B), 64, 0, st>>>(a, nullptr, nullptr, seg);
  scan_fwd_kernel<1, T><<<dim3(nx, a.P, B), 64, 0, st>>>(a, (__nv_bfloat16*)out, ckpt, seg);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace kmoe

using namespace kmoe;

extern "C" long long kmoe_scan_ckpt_floats(int B, int S, int C) {
  return (long long)B * ((S + CK - 1) / CK) * ((C + WCH - 1) / WCH) * (WCH * SN);
}

extern "C" int kmoe_scan_segments(int B, int S, int C) {
  int P, len;
  plan(B, S, C, &P, &len);
  return P;
}

extern "C" int kmoe_scan_fwd(const void* u, const void* delta, const void* z, const float* A, const void* Bm,
                             const void* Cm, long long ldbc, int bc_bf16, const float* D, const float* dt_bias, void* out,
                             float* ckpt, float* seg, int B, int S, int C, int N, long long ldz, int softplus, int groups,
                             cudaStream_t st) {
  ScanArgs a{(const __nv_bfloat16*)u, (const __nv_bfloat16*)delta, (const __nv_bfloat16*)z, A, Bm, Cm, D, dt_bias,
             S, C, ldz, ldbc, softplus, groups > 0 ? B / groups : 0, 1, 0};
  if (int rc = kmoe::check(a, bc_bf16, B, N, groups)) return rc;
  if (B == 0 || S == 0 || C == 0) return 0;    // the kernels need a chunk: their warps finish one after the last
  plan(B, S, C, &a.P, &a.seg_len);
  if (a.P > 1 && seg == nullptr) return -5;
  return bc_bf16 ? launch_fwd<__nv_bfloat16>(a, out, ckpt, seg, B, st) : launch_fwd<float>(a, out, ckpt, seg, B, st);
}

// dA [G,C,N], dB/dC [B,S,N], dD [G,C], dbias [G,C] (G = groups) are fp32 and must be zeroed by the caller.
// seg: the forward's segment scratch; gseg: scratch of B * P * C * N floats.
extern "C" int kmoe_scan_bwd(const void* u, const void* delta, const void* z, const float* A, const void* Bm,
                             const void* Cm, long long ldbc, int bc_bf16, const float* D, const float* dt_bias,
                             const void* dout, const float* ckpt, const float* seg, float* gseg, void* du, void* ddelta,
                             void* dz, long long lddz, float* dA, float* dB, float* dC, float* dD, float* dbias, int B,
                             int S, int C, int N, long long ldz, int softplus, int groups, cudaStream_t st) {
  ScanArgs a{(const __nv_bfloat16*)u, (const __nv_bfloat16*)delta, (const __nv_bfloat16*)z, A, Bm, Cm, D, dt_bias,
             S, C, ldz, ldbc, softplus, groups > 0 ? B / groups : 0, 1, 0};
  if (int rc = kmoe::check(a, bc_bf16, B, N, groups)) return rc;
  if (z != nullptr && lddz % 8) return -4;
  if (B == 0 || S == 0 || C == 0) return 0;    // as above; the sums stay at the caller's zeros
  plan(B, S, C, &a.P, &a.seg_len);
  if (a.P > 1 && (seg == nullptr || gseg == nullptr)) return -5;
  const int nx = (C + WCH - 1) / WCH;
  const __nv_bfloat16* go = (const __nv_bfloat16*)dout;
  auto carry = bc_bf16 ? scan_bwd_carry_kernel<__nv_bfloat16> : scan_bwd_carry_kernel<float>;
  auto bwd = bc_bf16 ? scan_bwd_kernel<__nv_bfloat16> : scan_bwd_kernel<float>;
  if (a.P > 1) carry<<<dim3(nx, a.P - 1, B), 64, 0, st>>>(a, go, gseg);
  bwd<<<dim3(nx, a.P, B), 64, 0, st>>>(a, go, ckpt, seg, gseg, (__nv_bfloat16*)du, (__nv_bfloat16*)ddelta,
                                       (__nv_bfloat16*)dz, lddz, dA, dB, dC, dD, dbias);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
