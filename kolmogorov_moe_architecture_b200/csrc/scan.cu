// Selective scan (Mamba), forward and backward, channels-last bf16 activations.
//
//   h_t[n] = exp(dt_t A[n]) h_{t-1}[n] + dt_t u_t B_t[n]        y_t = sum_n C_t[n] h_t[n] + D u_t   (* silu(z_t))
//
// Layout of the work: four lanes share a channel and keep four of its N = 16 states each, in registers, as two packed
// fp32 pairs; a warp owns 8 channels (lane = channel + 8 * state group) and walks the sequence in chunks of 8 steps
// without waiting for the CTA's other warps: it copies its own inputs (cp.async, one 16-byte piece per lane, array and
// step), prepares what a step needs once per channel (softplus, gates, products; two (step, channel) pairs per lane),
// then carries the recurrence.  Sums over the states of a channel meet in three shuffles per four steps: each lane ends
// up owning one of the steps and finishes it.
// With 4 x 4096 channels this fills the chip with one pass over the sequence.  Fewer channels are cut into P segments
// that run in parallel (the recurrence is linear, so a segment started from zero only lacks
// decay(segment) * state_before):
//   forward : pass 1 computes each segment's end state from zero and its sum of dt; pass 2 starts every segment
//             from the true state (a short serial combination of the earlier segments) and writes y plus a
//             state checkpoint every 8 steps.
//   backward: pass 1 runs dL/dh backwards through each segment from zero; pass 2 starts from the true incoming
//             value, replays a chunk from its checkpoint - decays and states stay in registers - and walks it in reverse.
// dB and dC are sums over channels: a warp lays four steps of its lanes' values out in shared memory and each lane adds up
// eight 16-byte pieces; the CTA's warps meet once per chunk, CTAs in 16-byte global reductions.
//
// Bounds: issue slots.  The 16 exponentials per channel and step alone take 119 us per pass of 4 x 2048 x 4096 on the
// MUFU pipe; the instructions around them (backward: about a third each for the packed arithmetic, the two kinds of sums,
// and operand reads with the per-channel preparation) take more: 4 x 2048 x 4096 forward 344 us, backward 831 us, at
// 60 - 65 % of the issue slots.  One thread per channel with all 16 states, which this replaces, needed two passes in each
// direction to fill the chip (147 + 223 and 160 + 1029 us); 1 x 333 x 1536 took 116 us in all, now 48.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kmoe_api.h"
#include "ptx.cuh"

namespace kmoe {

constexpr int SN = 16;        // states
constexpr int CK = 8;         // checkpoint interval = steps per chunk
constexpr int WCH = 8;        // channels per warp
constexpr int SW = 2;         // warps per CTA: few, so that CTAs of equal length fill the SMs evenly
constexpr int SCH = SW * WCH; // channels per CTA
constexpr int STH = SW * 32;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

__device__ __forceinline__ float s_bf2f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float s_softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }
__device__ __forceinline__ float s_sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }
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
// four values of B or C as two packed pairs
__device__ __forceinline__ void s_load4(const float* p, uint64_t (&v)[2]) {
  const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(p);
  v[0] = q.x;
  v[1] = q.y;
}
__device__ __forceinline__ void s_load4(const __nv_bfloat16* p, uint64_t (&v)[2]) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  v[0] = pack_f32x2(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xffff0000u));
  v[1] = pack_f32x2(__uint_as_float(q.y << 16), __uint_as_float(q.y & 0xffff0000u));
}
__device__ __forceinline__ float4 s_unpack4(const uint64_t (&v)[2]) {
  float4 q;
  unpack_f32x2(v[0], q.x, q.y);
  unpack_f32x2(v[1], q.z, q.w);
  return q;
}
// x[s] of four steps, summed over the four state groups (lane bits 3 and 4): lane group k returns the sum of step k
__device__ __forceinline__ float s_sum_states(const float (&x)[4], int sg) {
  const bool hi = sg & 2, odd = sg & 1;
  const float k0 = hi ? x[2] : x[0], k1 = hi ? x[3] : x[1], g0 = hi ? x[0] : x[2], g1 = hi ? x[1] : x[3];
  const float y0 = k0 + __shfl_xor_sync(0xffffffffu, g0, 16), y1 = k1 + __shfl_xor_sync(0xffffffffu, g1, 16);
  return (odd ? y1 : y0) + __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 8);
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

// Inputs of one chunk of one warp.  T: element type of B and C.
template <typename T>
struct __align__(16) RawTile {
  __nv_bfloat16 x[4][CK][WCH];                 // which four arrays is the kernel's business
  T bc[2][CK][SN];
};
// Staging of a chunk: a lane copies one 16-byte piece (array lane / 8, step lane % 8) and one or two pieces of B and C.
// Its sources never change, only the step does.
template <typename T>
struct Feeder {
  static constexpr int PIECES = SN * (int)sizeof(T) / 16;      // of a row of B or C
  static constexpr int PER_LANE = 2 * CK * PIECES / 32;
  const __nv_bfloat16* src;    // this lane's array at step 0 of the batch entry; null = nothing to copy
  long long ld;
  const T *Bm, *Cm;            // rows of the batch entry; null = not wanted
  __device__ __forceinline__ Feeder(const ScanArgs& a, const __nv_bfloat16* s0, long long l0, const __nv_bfloat16* s1,
                                    long long l1, const __nv_bfloat16* s2, long long l2, const __nv_bfloat16* s3,
                                    long long l3, bool wantB, bool wantC, int b, int cw, int lane) {
    const int k = lane >> 3;
    src = k == 0 ? s0 : (k == 1 ? s1 : (k == 2 ? s2 : s3));
    ld = k == 0 ? l0 : (k == 1 ? l1 : (k == 2 ? l2 : l3));
    if (src != nullptr) src += (size_t)b * a.S * ld + cw;
    Bm = wantB ? reinterpret_cast<const T*>(a.Bm) + (size_t)b * a.S * a.ldbc : nullptr;
    Cm = wantC ? reinterpret_cast<const T*>(a.Cm) + (size_t)b * a.S * a.ldbc : nullptr;
  }
  __device__ __forceinline__ void load(RawTile<T>& st, const ScanArgs& a, int t0, int t_end, bool live, int lane) const {
    const int row = lane & 7, t = t0 + row;
    if (src != nullptr)
      s_cp16(&st.x[lane >> 3][row][0], src + (size_t)(t < t_end ? t : t_end - 1) * ld, live && t < t_end);
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int j = lane + 32 * i, which = j / (CK * PIECES), r2 = (j / PIECES) % CK, pt = j % PIECES, t2 = t0 + r2;
      const T* base = which ? Cm : Bm;
      if (base != nullptr)
        s_cp16(&st.bc[which][r2][pt * (16 / (int)sizeof(T))],
               base + (size_t)(t2 < t_end ? t2 : t_end - 1) * a.ldbc + pt * (16 / (int)sizeof(T)), t2 < t_end);
    }
    s_commit();
  }
};

// MODE 0: end state from zero + sum of dt (segments 0 .. P-2).  MODE 1: outputs and checkpoints.
template <int MODE, typename T>
__global__ void __launch_bounds__(STH)
scan_fwd_kernel(ScanArgs a, __nv_bfloat16* __restrict__ out, float* __restrict__ ckpt, float* __restrict__ seg) {
  struct __align__(16) Warp {
    RawTile<T> st[2];
    float2 sc[CK][WCH];                        // dt, dt * u
    float2 so[CK][WCH];                        // D * u, gate
    __nv_bfloat16 y[CK][WCH];
  };
  __shared__ Warp warps[SW];
  const int tid = threadIdx.x, lane = tid & 31, ch = lane & 7, sg = lane >> 3;
  Warp& w = warps[tid >> 5];
  const int cw = blockIdx.x * SCH + (tid >> 5) * WCH, c = cw + ch, p = blockIdx.y, b = blockIdx.z;
  if (cw >= a.C) return;                       // C is a multiple of 8: a warp's channels exist or do not, together
  const int pc = (b / a.bpg) * a.C + c;
  const bool has_z = a.z != nullptr;
  const int t_begin = p * a.seg_len, t_end = min(a.S, t_begin + a.seg_len);
  const size_t nrows = (size_t)gridDim.z * a.P * a.C;      // rows of the segment scratch
  uint64_t An[2], h[2];
  {
    const float4 v = *reinterpret_cast<const float4*>(a.A + (size_t)pc * SN + sg * 4);
    An[0] = pack_f32x2(v.x * LOG2E, v.y * LOG2E);
    An[1] = pack_f32x2(v.z * LOG2E, v.w * LOG2E);
    h[0] = h[1] = s_dup(0.f);
  }
  if (MODE == 1) {
    // state before this segment: fold the earlier segments' zero-started end states, oldest first
    for (int q = 0; q < p; ++q) {
      const size_t r = seg_row(a, b, q, c);
      const uint64_t sdt = s_dup(seg[nrows * SN + r]);
      const float4 e = *reinterpret_cast<const float4*>(seg + r * SN + sg * 4);
      h[0] = fma_f32x2(s_ex2x2(mul_f32x2(An[0], sdt)), h[0], pack_f32x2(e.x, e.y));
      h[1] = fma_f32x2(s_ex2x2(mul_f32x2(An[1], sdt)), h[1], pack_f32x2(e.z, e.w));
    }
  }
  const float Dc = a.D ? a.D[pc] : 0.f, bias = a.dt_bias ? a.dt_bias[pc] : 0.f;
  float sdt = 0.f;
  const int nchunks = (a.S + CK - 1) / CK;
  const int ntiles = (t_end - t_begin + CK - 1) / CK;
  const Feeder<T> feed(a, a.u, a.C, a.delta, a.C, MODE == 1 ? a.z : nullptr, a.ldz, nullptr, 0, true, MODE == 1, b, cw,
                       lane);
  float* ck = (MODE == 1 && ckpt != nullptr) ? ckpt + (((size_t)b * nchunks + t_begin / CK) * a.C + c) * SN + sg * 4 : nullptr;

  feed.load(w.st[0], a, t_begin, t_end, true, lane);
  for (int tile = 0; tile < ntiles; ++tile) {
    const RawTile<T>& st = w.st[tile & 1];
    const int t0 = t_begin + tile * CK;
    s_wait<0>();
    __syncwarp();                              // this chunk has landed; every lane is done with the previous one
    if (tile + 1 < ntiles) feed.load(w.st[(tile + 1) & 1], a, t0 + CK, t_end, true, lane);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int row = sg + 4 * k;
      const bool ok = t0 + row < t_end;        // steps past the end leave the state alone
      const float uu = s_bf2f(st.x[0][row][ch]);
      float dt = s_bf2f(st.x[1][row][ch]) + bias;
      if (a.softplus) dt = s_softplus(dt);
      if (!ok) dt = 0.f;
      w.sc[row][ch] = make_float2(dt, dt * uu);
      if (MODE == 1) {
        float gate = 1.f;
        if (has_z) {
          const float zv = s_bf2f(st.x[2][row][ch]);
          gate = zv * s_sigmoid(zv);
        }
        w.so[row][ch] = make_float2(Dc * uu, gate);
      }
    }
    if (MODE == 1 && ck != nullptr) {
      *reinterpret_cast<float4*>(ck) = s_unpack4(h);
      ck += (size_t)a.C * SN;
    }
    __syncwarp();
    // no store to shared memory before the chunk's last read: it would keep the reads of later steps behind it
    float yv[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float ys[4];
#pragma unroll
      for (int i4 = 0; i4 < 4; ++i4) {
        const int i = half * 4 + i4;
        const float2 d = w.sc[i][ch];
        uint64_t Bv[2];
        s_load4(&st.bc[0][i][sg * 4], Bv);
        const uint64_t dt2 = s_dup(d.x), dtu2 = s_dup(d.y);
        h[0] = fma_f32x2(s_ex2x2(mul_f32x2(dt2, An[0])), h[0], mul_f32x2(dtu2, Bv[0]));
        h[1] = fma_f32x2(s_ex2x2(mul_f32x2(dt2, An[1])), h[1], mul_f32x2(dtu2, Bv[1]));
        if (MODE == 1) {
          uint64_t Cv[2];
          s_load4(&st.bc[1][i][sg * 4], Cv);
          ys[i4] = s_hsum(fma_f32x2(Cv[1], h[1], mul_f32x2(Cv[0], h[0])));
        } else {
          sdt += d.x;
        }
      }
      if (MODE == 1) {
        const float2 q = w.so[half * 4 + sg][ch];
        yv[half] = (s_sum_states(ys, sg) + q.x) * q.y;
      }
    }
    if (MODE == 1) {
      w.y[sg][ch] = __float2bfloat16(yv[0]);
      w.y[4 + sg][ch] = __float2bfloat16(yv[1]);
      __syncwarp();
      if (lane < CK && t0 + lane < t_end)
        *reinterpret_cast<uint4*>(out + ((size_t)b * a.S + t0 + lane) * a.C + cw) =
            *reinterpret_cast<const uint4*>(&w.y[lane][0]);
    }
  }
  if (MODE == 0) {
    const size_t r = seg_row(a, b, p, c);
    *reinterpret_cast<float4*>(seg + r * SN + sg * 4) = s_unpack4(h);
    if (sg == 0) seg[nrows * SN + r] = sdt;
  }
}

// ------------------------------------------------------------------ backward, pass 1
// dL/dh carried backwards through segment p (1 .. P-1) from zero: gseg[b][p][c][n] = what the segment hands to
// the step before its first one.
template <typename T>
__global__ void __launch_bounds__(STH)
scan_bwd_carry_kernel(ScanArgs a, const __nv_bfloat16* __restrict__ dout, float* __restrict__ gseg) {
  struct __align__(16) Warp {
    RawTile<T> st[2];
    float2 sc[CK][WCH];                        // dt, dL/dy
  };
  __shared__ Warp warps[SW];
  const int tid = threadIdx.x, lane = tid & 31, ch = lane & 7, sg = lane >> 3;
  Warp& w = warps[tid >> 5];
  const int cw = blockIdx.x * SCH + (tid >> 5) * WCH, c = cw + ch, p = blockIdx.y + 1, b = blockIdx.z;
  if (cw >= a.C) return;
  const int pc = (b / a.bpg) * a.C + c;
  const bool has_z = a.z != nullptr;
  const int t_begin = p * a.seg_len, t_end = min(a.S, t_begin + a.seg_len);
  uint64_t An[2], g[2];
  {
    const float4 v = *reinterpret_cast<const float4*>(a.A + (size_t)pc * SN + sg * 4);
    An[0] = pack_f32x2(v.x * LOG2E, v.y * LOG2E);
    An[1] = pack_f32x2(v.z * LOG2E, v.w * LOG2E);
    g[0] = g[1] = s_dup(0.f);
  }
  const float bias = a.dt_bias ? a.dt_bias[pc] : 0.f;
  const int ntiles = (t_end - t_begin + CK - 1) / CK;
  const Feeder<T> feed(a, a.delta, a.C, a.z, a.ldz, dout, a.C, nullptr, 0, false, true, b, cw, lane);
  feed.load(w.st[0], a, t_begin + (ntiles - 1) * CK, t_end, true, lane);
  int s = 0;
  for (int tile = ntiles - 1; tile >= 0; --tile, s ^= 1) {
    const RawTile<T>& st = w.st[s];
    const int t0 = t_begin + tile * CK;
    s_wait<0>();
    __syncwarp();
    if (tile > 0) feed.load(w.st[s ^ 1], a, t0 - CK, t_end, true, lane);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int row = sg + 4 * k;
      float dt = s_bf2f(st.x[0][row][ch]) + bias;
      if (a.softplus) dt = s_softplus(dt);
      float dy = s_bf2f(st.x[2][row][ch]);
      if (has_z) {
        const float zv = s_bf2f(st.x[1][row][ch]);
        dy *= zv * s_sigmoid(zv);
      }
      w.sc[row][ch] = t0 + row < t_end ? make_float2(dt, dy) : make_float2(0.f, 0.f);
    }
    __syncwarp();
#pragma unroll
    for (int i = CK - 1; i >= 0; --i) {
      const float2 d = w.sc[i][ch];
      uint64_t Cv[2];
      s_load4(&st.bc[1][i][sg * 4], Cv);
      const uint64_t dt2 = s_dup(d.x), dy2 = s_dup(d.y);
      g[0] = mul_f32x2(fma_f32x2(Cv[0], dy2, g[0]), s_ex2x2(mul_f32x2(dt2, An[0])));
      g[1] = mul_f32x2(fma_f32x2(Cv[1], dy2, g[1]), s_ex2x2(mul_f32x2(dt2, An[1])));
    }
  }
  *reinterpret_cast<float4*>(gseg + seg_row(a, b, p, c) * SN + sg * 4) = s_unpack4(g);
}

// ------------------------------------------------------------------ backward, pass 2
template <typename T>
__global__ void __launch_bounds__(STH, 8)
scan_bwd_kernel(ScanArgs a, const __nv_bfloat16* __restrict__ dout, const float* __restrict__ ckpt,
                const float* __restrict__ seg, const float* __restrict__ gseg, __nv_bfloat16* __restrict__ du,
                __nv_bfloat16* __restrict__ ddelta, __nv_bfloat16* __restrict__ dz, long long lddz,
                float* __restrict__ dA, float* __restrict__ dB, float* __restrict__ dC, float* __restrict__ dD,
                float* __restrict__ dbias) {
  struct __align__(16) Warp {
    RawTile<T> st[2];                          // u, delta, z, dout
    float4 sc[CK][WCH];                        // dt, dt * u, dL/dy, u
    float2 sd[CK][WCH];                        // dz / y factor, softplus'
    __nv_bfloat16 o[3][CK][WCH];               // du, ddelta, dz
    float4 part[4][2][32];                     // four steps of every lane's dB and dC, to be summed over the channels
    float red[2][CK][2 * SN];                  // the warp's channel sums of dB and dC, by chunk parity
  };
  __shared__ Warp warps[SW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ch = lane & 7, sg = lane >> 3;
  Warp& w = warps[warp];
  const int cw = blockIdx.x * SCH + warp * WCH, p = blockIdx.y, b = blockIdx.z;
  const bool live = cw < a.C;                  // a warp without channels computes on zeros and stores nothing
  const int c = (live ? cw : 0) + ch;
  const int pc = (b / a.bpg) * a.C + c;
  const bool has_z = a.z != nullptr;
  const int t_begin = p * a.seg_len, t_end = min(a.S, t_begin + a.seg_len);
  const size_t nrows = (size_t)gridDim.z * a.P * a.C;
  uint64_t An[2], g[2], dAacc[2];
  {
    const float4 v = *reinterpret_cast<const float4*>(a.A + (size_t)pc * SN + sg * 4);
    An[0] = pack_f32x2(v.x * LOG2E, v.y * LOG2E);
    An[1] = pack_f32x2(v.z * LOG2E, v.w * LOG2E);
    g[0] = g[1] = dAacc[0] = dAacc[1] = s_dup(0.f);
  }
  // dL/dh flowing into the last step of this segment: fold the later segments' zero-started carries, last first
  for (int q = a.P - 1; q > p; --q) {
    const size_t r = seg_row(a, b, q, c);
    const uint64_t sdt = s_dup((q < a.P - 1) ? seg[nrows * SN + r] : 0.f);
    const float4 e = *reinterpret_cast<const float4*>(gseg + r * SN + sg * 4);
    g[0] = fma_f32x2(s_ex2x2(mul_f32x2(An[0], sdt)), g[0], pack_f32x2(e.x, e.y));
    g[1] = fma_f32x2(s_ex2x2(mul_f32x2(An[1], sdt)), g[1], pack_f32x2(e.z, e.w));
  }
  const float Dc = a.D ? a.D[pc] : 0.f, bias = a.dt_bias ? a.dt_bias[pc] : 0.f;
  float dDacc = 0.f, dbacc = 0.f;
  const int nchunks = (a.S + CK - 1) / CK;
  const int ntiles = (t_end - t_begin + CK - 1) / CK;
  const Feeder<T> feed(a, a.u, a.C, a.delta, a.C, a.z, a.ldz, dout, a.C, true, true, b, live ? cw : 0, lane);
  const float* ck = ckpt + (((size_t)b * nchunks + t_begin / CK + ntiles - 1) * a.C + c) * SN + sg * 4;

  feed.load(w.st[0], a, t_begin + (ntiles - 1) * CK, t_end, live, lane);
  float4 hn = __ldg(reinterpret_cast<const float4*>(ck));
  int s = 0;
  for (int tile = ntiles - 1; tile >= 0; --tile, s ^= 1) {
    const RawTile<T>& st = w.st[s];
    const int t0 = t_begin + tile * CK;
    const uint64_t h0[2] = {pack_f32x2(hn.x, hn.y), pack_f32x2(hn.z, hn.w)};
    s_wait<0>();
    __syncwarp();
    if (tile > 0) {
      feed.load(w.st[s ^ 1], a, t0 - CK, t_end, live, lane);
      ck -= (size_t)a.C * SN;
      hn = __ldg(reinterpret_cast<const float4*>(ck));     // in flight while this chunk is processed
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int row = sg + 4 * k;
      const bool ok = live && t0 + row < t_end;            // steps past the end: decay 1, nothing added, nothing summed
      const float uu = s_bf2f(st.x[0][row][ch]);
      const float dtr = s_bf2f(st.x[1][row][ch]) + bias;
      const float dt = a.softplus ? s_softplus(dtr) : dtr;
      float dy = s_bf2f(st.x[3][row][ch]), zf = 0.f;
      if (has_z) {
        const float zv = s_bf2f(st.x[2][row][ch]);
        const float sgm = s_sigmoid(zv);
        zf = dy * sgm * (1.f + zv * (1.f - sgm));
        dy *= zv * sgm;
      }
      w.sc[row][ch] = ok ? make_float4(dt, dt * uu, dy, uu) : make_float4(0.f, 0.f, 0.f, 0.f);
      w.sd[row][ch] = ok ? make_float2(zf, a.softplus ? s_sigmoid(dtr) : 1.f) : make_float2(0.f, 0.f);
    }
    __syncwarp();
    // replay the chunk forward: decay of every step and state after it
    uint64_t an[CK][2], h[CK][2];
#pragma unroll
    for (int i = 0; i < CK; ++i) {
      const float2 d = *reinterpret_cast<const float2*>(&w.sc[i][ch]);
      uint64_t Bv[2];
      s_load4(&st.bc[0][i][sg * 4], Bv);
      const uint64_t dt2 = s_dup(d.x), dtu2 = s_dup(d.y);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        an[i][k] = s_ex2x2(mul_f32x2(dt2, An[k]));
        h[i][k] = fma_f32x2(an[i][k], i > 0 ? h[i - 1][k] : h0[k], mul_f32x2(dtu2, Bv[k]));
      }
    }
    // reverse sweep
#pragma unroll
    for (int half = 1; half >= 0; --half) {
      float sA[4], sB[4], yp[4];               // sums over this lane's states of the half's four steps
#pragma unroll
      for (int i4 = 3; i4 >= 0; --i4) {
        const int i = half * 4 + i4;
        const float4 d = w.sc[i][ch];
        const uint64_t dt2 = s_dup(d.x), dtu2 = s_dup(d.y), dy2 = s_dup(d.z);
        uint64_t Bv[2], Cv[2];
        s_load4(&st.bc[0][i][sg * 4], Bv);
        s_load4(&st.bc[1][i][sg * 4], Cv);
        uint64_t a2, b2, y2;
        ulonglong2 vB, vC;                     // dB and dC of the lane's four states
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          y2 = k == 0 ? mul_f32x2(Cv[k], h[i][k]) : fma_f32x2(Cv[k], h[i][k], y2);
          (k == 0 ? vC.x : vC.y) = mul_f32x2(dy2, h[i][k]);
          const uint64_t gn = fma_f32x2(Cv[k], dy2, g[k]);               // dL/dh_t
          b2 = k == 0 ? mul_f32x2(gn, Bv[k]) : fma_f32x2(gn, Bv[k], b2);
          (k == 0 ? vB.x : vB.y) = mul_f32x2(gn, dtu2);
          g[k] = mul_f32x2(gn, an[i][k]);                                // handed to step t - 1
          const uint64_t gh = mul_f32x2(g[k], i > 0 ? h[i - 1][k] : h0[k]);
          a2 = k == 0 ? mul_f32x2(gh, An[k]) : fma_f32x2(gh, An[k], a2);
          dAacc[k] = fma_f32x2(gh, dt2, dAacc[k]);
        }
        *reinterpret_cast<ulonglong2*>(&w.part[i4][0][lane]) = vB;
        *reinterpret_cast<ulonglong2*>(&w.part[i4][1][lane]) = vC;
        sA[i4] = s_hsum(a2);
        sB[i4] = s_hsum(b2);
        yp[i4] = s_hsum(y2);
      }
      // this lane finishes step half * 4 + sg of its channel
      const float tA = s_sum_states(sA, sg), tB = s_sum_states(sB, sg), ty = s_sum_states(yp, sg);
      const float4 d = w.sc[half * 4 + sg][ch];
      const float2 e = w.sd[half * 4 + sg][ch];
      const float dd = (tA * LN2 + d.w * tB) * e.y;
      dDacc += d.z * d.w;
      dbacc += dd;
      w.o[0][half * 4 + sg][ch] = __float2bfloat16(d.x * tB + d.z * Dc);
      w.o[1][half * 4 + sg][ch] = __float2bfloat16(dd);
      w.o[2][half * 4 + sg][ch] = __float2bfloat16(e.x * (ty + Dc * d.w));
      // channel sums: this lane takes four values (dB or dC of state group lane & 3) of step lane / 8; the lanes of a
      // step start at different channels, which keeps their 16-byte reads on different banks
      __syncwarp();
      uint64_t acc[2] = {0, 0};
#pragma unroll
      for (int k = 0; k < WCH; ++k) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(
            &w.part[lane >> 3][(lane >> 2) & 1][(lane & 3) * 8 + ((k + lane) & 7)]);
        acc[0] = k == 0 ? q.x : add_f32x2(acc[0], q.x);
        acc[1] = k == 0 ? q.y : add_f32x2(acc[1], q.y);
      }
      *reinterpret_cast<ulonglong2*>(&w.red[s][half * 4 + (lane >> 3)][(lane & 7) * 4]) = make_ulonglong2(acc[0], acc[1]);
      __syncwarp();
    }
    // the warps' channel sums of this chunk are complete; those of the previous chunk (other parity) have been read
    __syncthreads();
    if (lane < 24) {
      const int k = lane >> 3, t = t0 + ch;
      if (live && t < t_end && (k < 2 || has_z)) {
        __nv_bfloat16* dst = k == 0 ? du : (k == 1 ? ddelta : dz);
        *reinterpret_cast<uint4*>(dst + ((size_t)b * a.S + t) * (k == 2 ? lddz : (long long)a.C) + cw) =
            *reinterpret_cast<const uint4*>(&w.o[k][ch][0]);
      }
    }
    {
      const int row = warp * (CK / SW) + sg, quad = ch, t = t0 + row;
      float4 v = *reinterpret_cast<const float4*>(&warps[0].red[s][row][quad * 4]);
#pragma unroll
      for (int k = 1; k < SW; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(&warps[k].red[s][row][quad * 4]);
        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
      }
      if (t < t_end) s_red4((quad < 4 ? dB : dC) + ((size_t)b * a.S + t) * SN + (quad & 3) * 4, v);
    }
  }
#pragma unroll
  for (int k = 8; k <= 16; k <<= 1) {
    dDacc += __shfl_xor_sync(0xffffffffu, dDacc, k);
    dbacc += __shfl_xor_sync(0xffffffffu, dbacc, k);
  }
  if (live) {
    s_red4(dA + (size_t)pc * SN + sg * 4, s_unpack4(dAacc));
    if (sg == 0 && dD) atomicAdd(&dD[pc], dDacc);
    if (sg == 0 && dbias) atomicAdd(&dbias[pc], dbacc);
  }
}
static_assert(SW * 4 == CK, "a warp flushes four steps of the channel sums");

// Segment count: the one that minimises (rounds of CTAs per SM) x (steps per segment).  Up to about four CTAs on an
// SM the time of a step is its latency, beyond that it grows with the CTAs; cutting the sequence at all costs a second
// pass over it (about half of the work again).  Forward + backward of 1 x 2048 x 4096 in one segment 670 us, in four 382.
// Segments are multiples of the chunk and at least 64 steps long.
static void plan(int B, int S, int C, int* P, int* seg_len) {
  const long long per_seg = (long long)((C + SCH - 1) / SCH) * B;
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
  const int nx = (a.C + SCH - 1) / SCH;
  if (a.P > 1) scan_fwd_kernel<0, T><<<dim3(nx, a.P - 1, B), STH, 0, st>>>(a, nullptr, nullptr, seg);
  scan_fwd_kernel<1, T><<<dim3(nx, a.P, B), STH, 0, st>>>(a, (__nv_bfloat16*)out, ckpt, seg);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace kmoe

using namespace kmoe;

extern "C" int kmoe_scan_chunk(void) { return CK; }

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
  plan(B, S, C, &a.P, &a.seg_len);
  if (a.P > 1 && (seg == nullptr || gseg == nullptr)) return -5;
  const int nx = (C + SCH - 1) / SCH;
  const __nv_bfloat16* go = (const __nv_bfloat16*)dout;
  auto carry = bc_bf16 ? scan_bwd_carry_kernel<__nv_bfloat16> : scan_bwd_carry_kernel<float>;
  auto bwd = bc_bf16 ? scan_bwd_kernel<__nv_bfloat16> : scan_bwd_kernel<float>;
  if (a.P > 1) carry<<<dim3(nx, a.P - 1, B), STH, 0, st>>>(a, go, gseg);
  bwd<<<dim3(nx, a.P, B), STH, 0, st>>>(a, go, ckpt, seg, gseg, (__nv_bfloat16*)du, (__nv_bfloat16*)ddelta,
                                        (__nv_bfloat16*)dz, lddz, dA, dB, dC, dD, dbias);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
