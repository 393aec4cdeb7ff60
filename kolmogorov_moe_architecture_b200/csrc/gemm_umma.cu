// Persistent warp-specialised bf16 GEMM for sm_100a.
//
//   warp 0      : TMA producer  (cp.async.bulk.tensor -> 128B-swizzled smem ring, mbarrier tx counts)
//   warp 1      : MMA issuer    (tcgen05.mma 128 x BN x 16, accumulators in TMEM, double buffered)
//   warps 2..5  : epilogue      (tcgen05.ld -> registers -> fused epilogue -> global); with eight of them warps 4..11
//
// One CTA per SM walks a static tile list, so the epilogue of tile i overlaps the
// main loop of tile i+1.  Operands may be K-major or MN-major (the MMA reads either
// from swizzled smem), which covers forward, dgrad and wgrad without transposes.
// Three tile schedules: dense, grouped along M (expert-sorted rows padded to 128
// per expert, tile->expert table and live tile count read from device memory: no
// host synchronisation), and batched (independent GEMMs, optionally with a ragged
// reduction range per group: the wgrad of the experts).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>

#include "kmoe_api.h"
#include "ptx.cuh"
#include "tmap_host.h"

namespace kmoe {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int A_STAGE_BYTES = BM * BK * 2;
// Four epilogue warps: 192 threads, and every thread has the registers it wants.
// Eight (CTA pairs with short reductions, see WIDE_K_PLAIN): three warpgroups, producer and issuer (and two idle warps), two of
// epilogue.  The registers, 384 x 168 at launch, are split unevenly, once: an increase waits without a limit for what
// others give up.  Handed back at the end, they could go round in a pair without a tile: its load and MMA warps took back
// what the epilogue warps were still waiting for.
constexpr int threads_of(int epi_warps) { return epi_warps == 8 ? 384 : 192; }
constexpr int CTA_EPI_WARPS = 4;
constexpr int LAUNCH_REGS = 168, EPI_REGS = 216, ROLE_REGS = 72;
static_assert(256 * EPI_REGS + 128 * ROLE_REGS == threads_of(8) * LAUNCH_REGS, "register split");
template <int N>
__device__ __forceinline__ void set_regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void set_regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

struct GemmArgs {
  void* C;
  const void* D;
  const void* D2;
  void* G_out;
  void* U_out;
  int mode, epilogue;
  int M, N, K, groups;
  long long ldc, ldd, c_gstride;
  int a_grouped, b_grouped;
  const int* tile_group;
  const int* num_m_tiles;
  const int* k_begin;
  const int* k_len;
  int out_f32;
  float alpha, beta, beta2;
  const float* row_scale;
  const float* alpha_dev;     // optional per-group multipliers of alpha / beta (BATCHED: index = group)
  const float* beta_dev;
  int sym_upper;              // C is symmetric (A == B): compute only tiles that touch the upper triangle
  float diag_add;             // added to C[i][i] after alpha (bf16 store path)
  int k_split;                // > 0: reduction elements [k_split, K) of B come from the second tensor map
  int a_boxed, b_boxed;       // MN-major operand whose row count is no multiple of 64: one 64-row box per load
  const long long* row_ptr;   // optional: address of each output row (may be peer memory); 0 = row not stored
  int* status;
};

// Reduction ranges of the first groups in shared memory: every role looks up its tiles' ranges one after the other, and
// from global memory that is 700 clocks each time.
constexpr int RANGES_MAX = 128;
__device__ __forceinline__ void fill_ranges(const GemmArgs& a, int2* ranges) {
  if (a.mode == KMOE_GEMM_BATCHED && a.k_begin != nullptr)
    for (int g = threadIdx.x; g < min(a.groups, RANGES_MAX); g += blockDim.x) ranges[g] = make_int2(a.k_begin[g], a.k_len[g]);
}

struct Tile {
  int m_tile, n_tile, g_a, g_b, g_c, k0, k_blocks;
  int row;        // first output row
  int rows_ok;    // CTA pair on the expert-padded schedule: 0 = the lower 128 rows belong to the next expert
};

// CTA pairs on the expert-padded schedule: two consecutive 128-row blocks of one expert make a 256-row tile, the last
// block of an expert with an odd count a tile of which only the upper half is stored.  list[i] = first block of tile i,
// bit 15 set when the second block is the same expert's.  Built by one warp of each CTA from the block -> expert table
// (four loads in flight per lane), returns the number of tiles.
constexpr int PAIR_LIST_MAX = 768;
__device__ __forceinline__ int build_pair_list(const int* __restrict__ tile_group, int blocks, uint16_t* list, int lane) {
  int tiles = 0, run = 0, prev = -1;                 // carried: first block of the current run, its expert
  for (int base = 0; base < blocks; base += 128) {
    int g[4], nx[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = base + j * 32 + lane;
      g[j] = b < blocks ? __ldg(tile_group + b) : -2;
      nx[j] = b + 1 < blocks ? __ldg(tile_group + b + 1) : -2;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = base + j * 32 + lane;
      int before = __shfl_up_sync(0xffffffffu, g[j], 1);
      if (lane == 0) before = prev;
      const uint32_t starts = __ballot_sync(0xffffffffu, g[j] != before);
      const uint32_t upto = starts & (0xffffffffu >> (31 - lane));
      const int my_run = upto ? base + j * 32 + 31 - __clz(upto) : run;
      const bool first = b < blocks && ((b - my_run) & 1) == 0;
      const uint32_t emit = __ballot_sync(0xffffffffu, first);
      if (first) list[tiles + __popc(emit & ((1u << lane) - 1))] = (uint16_t)(b | (nx[j] == g[j] ? 0x8000 : 0));
      tiles += __popc(emit);
      run = __shfl_sync(0xffffffffu, my_run, 31);
      prev = __shfl_sync(0xffffffffu, g[j], 31);
    }
  }
  return tiles;
}

__device__ __forceinline__ int ceil_div(int a, int b) { return (a + b - 1) / b; }

// a / d for the small non-negative numbers of a tile list: a float quotient put right by one.  The compiler's division is
// about five times as long, and every role takes several per tile, one after the other.
__device__ __forceinline__ int list_div(int a, int d) {
  if (a >= 1 << 21) return a / d;           // __fdividef is good to two units in the last place: less than one here
  const int q = (int)__fdividef((float)a, (float)d), r = a - q * d;
  return q + (r >= d ? 1 : 0) - (r < 0 ? 1 : 0);
}

// Maps a linear work index to a tile of TM x BN outputs. Returns false past the end.
template <int BN, int TM = BM>
__device__ __forceinline__ bool get_tile(const GemmArgs& a, int idx, int num_m, int num_n, Tile& t, const int2* ranges,
                                         const uint16_t* pair_list = nullptr) {
  const int n_out = (a.epilogue == KMOE_EPI_SWIGLU) ? BN / 2 : BN;
  (void)n_out;
  int per_group = num_m * num_n;
  int g = 0, local = idx;
  if (a.sym_upper) {
    // enumerate only the tiles that touch the upper triangle, row by row, so that the work is spread evenly
    int kept = 0;
    for (int m = 0; m < num_m; ++m) kept += num_n - min(num_n, (m * TM) / BN);
    g = list_div(idx, kept);
    local = idx - g * kept;
    if (g >= (a.mode == KMOE_GEMM_BATCHED ? a.groups : 1)) return false;
    int m = 0;
    while (true) {
      const int km = num_n - min(num_n, (m * TM) / BN);
      if (local < km) break;
      local -= km;
      ++m;
    }
    t.m_tile = m;
    t.n_tile = min(num_n, (m * TM) / BN) + local;
  } else {
    if (a.mode == KMOE_GEMM_BATCHED) {
      g = list_div(idx, per_group);
      local = idx - g * per_group;
      if (g >= a.groups) return false;
    } else if (idx >= per_group) {
      return false;
    }
    // supertile of 8 m-tiles: neighbouring CTAs share B tiles and a narrow band of A
    const int GM = 8;
    int band = list_div(local, GM * num_n);
    int first_m = band * GM;
    int gsz = min(num_m - first_m, GM);
    int r = local - band * GM * num_n;
    t.n_tile = list_div(r, gsz);
    t.m_tile = first_m + r - t.n_tile * gsz;
  }
  t.k0 = 0;
  t.k_blocks = ceil_div(a.K, BK);
  t.row = t.m_tile * TM;
  t.rows_ok = 1;
  if (a.mode == KMOE_GEMM_GROUPED_M) {
    int block = t.m_tile;
    if (TM == 2 * BM) {
      const int entry = pair_list[t.m_tile];
      block = entry & 0x7fff;
      t.row = block * BM;
      t.rows_ok = entry >> 15;
    }
    int e = a.tile_group[block];
    t.g_a = 0;
    t.g_b = e;
    t.g_c = 0;
  } else if (a.mode == KMOE_GEMM_BATCHED) {
    t.g_a = a.a_grouped ? g : 0;
    t.g_b = a.b_grouped ? g : 0;
    t.g_c = g;
    if (a.k_begin != nullptr) {
      const int2 r = g < RANGES_MAX ? ranges[g] : make_int2(a.k_begin[g], a.k_len[g]);
      t.k0 = r.x;
      t.k_blocks = ceil_div(r.y, BK);
    }
  } else {
    t.g_a = t.g_b = t.g_c = 0;
  }
  return true;
}

template <typename T>
__device__ __forceinline__ void store8(T* dst, const float* v);
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16* dst, const float* v) {
  uint4 o;
  o.x = pack_bf16(v[0], v[1]);
  o.y = pack_bf16(v[2], v[3]);
  o.z = pack_bf16(v[4], v[5]);
  o.w = pack_bf16(v[6], v[7]);
  *reinterpret_cast<uint4*>(dst) = o;
}
template <>
__device__ __forceinline__ void store8<float>(float* dst, const float* v) {
  *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void load8(const __nv_bfloat16* src, float* v) {
  uint4 r = *reinterpret_cast<const uint4*>(src);
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(p[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load8(const float* src, float* v) {
  float4 a = *reinterpret_cast<const float4*>(src);
  float4 b = *reinterpret_cast<const float4*>(src + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// Writes one 32-column chunk of one fp32 row: out = scale * acc + beta * D
__device__ __forceinline__ void epilogue_store_chunk_f32(const GemmArgs& a, const uint32_t (&acc)[32], bool have_acc,
                                                         long long row_off_c, long long row_off_d, int col, float scale,
                                                         float beta) {
  float* C = reinterpret_cast<float*>(a.C);
  const float* D = reinterpret_cast<const float*>(a.D);
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    if (col + j >= a.N) break;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = have_acc ? __uint_as_float(acc[j + i]) * scale : 0.f;
    if (D != nullptr) {
      float d[8];
      load8(D + row_off_d + col + j, d);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] += beta * d[i];
    }
    store8<float>(C + row_off_c + col + j, v);
  }
}

// ------------------------------------------------------------------ bf16 epilogue
// An epilogue warp owns 32 accumulator rows (lane = row); of eight warps two share the rows, each with every other 64-column
// slab.  A slab is read from tensor memory, finished in registers, rounded into a 4 KB staging buffer (32 rows x 128 bytes
// in the 128-byte swizzle, so that both the row-per-lane writes and TMA's reads are free of bank conflicts) and sent off by
// a TMA store, which also clips at M and N.  One of four warps has two buffers, one of eight has one; it waits for a store
// to have read its buffer only when it has the values that go there next, and the accumulator goes back to the MMA warp
// as soon as the last slab is in registers.
// A tile whose reduction is shorter than its epilogue is bound by this code (weight gradients of experts with few tokens): a
// slab is a chain of latencies, so two warps per scheduler finish a tile sooner than one (see WIDE_K_PLAIN).
constexpr int OUT_BUF_BYTES = 32 * 128;
constexpr int OUT_STAGE_BYTES = 8 * OUT_BUF_BYTES;

template <int WARPS>
struct OutStage {
  static constexpr int STEP = WARPS / 4, BUFS = 8 / WARPS;
  uint8_t* base;   // of this warp's BUFS buffers
  int half;        // this warp's slabs: half, half + STEP, ...
  int buf;
  __device__ __forceinline__ OutStage(uint8_t* stage, int epi_warp)
      : base(stage + (WARPS == 4 ? epi_warp % 4 : epi_warp) * BUFS * OUT_BUF_BYTES),
        half(WARPS == 4 ? 0 : epi_warp / 4), buf(0) {}
};
template <int WARPS>
__device__ __forceinline__ uint8_t* out_acquire(OutStage<WARPS>& o, int lane) {
  if (lane == 0) {
    if (OutStage<WARPS>::BUFS == 2) tma_store_wait_read_but_one();
    else tma_store_wait_read();
  }
  __syncwarp();
  if (OutStage<WARPS>::BUFS == 1) return o.base;
  uint8_t* p = o.base + o.buf * OUT_BUF_BYTES;
  o.buf ^= 1;
  return p;
}
__device__ __forceinline__ void out_put_row(uint8_t* sb, int lane, const uint32_t (&p)[32]) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(sb + lane * 128 + ((j ^ (lane & 7)) << 4)) =
        make_uint4(p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
}
__device__ __forceinline__ void out_send(const CUtensorMap* tm, const uint8_t* sb, int lane, int x, int y, int g) {
  fence_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_store_4d(tm, sb, x, y, 0, g);
    tma_store_commit();
  }
}

// C = scale * acc (+ diag) (+ beta D + beta2 D2), all in fp32 before the one rounding.  `mirror`: the tile lies above
// the diagonal of a symmetric product and also writes its transpose (tmT: boxes of 32 columns x 64 rows).
// wait() returns once the accumulator is complete (false: gave up), release() hands it back.
template <int BN, class Stage, class Wait, class Release>
__device__ __forceinline__ bool store_tile_bf16(const GemmArgs& a, const CUtensorMap* tmC, const CUtensorMap* tmT,
                                                Stage& out, uint32_t t_row, bool have_acc, int row0, int n0, int g,
                                                float scale, float beta, float beta2, bool mirror, int lane,
                                                Wait wait, Release release) {
  const int slabs = row0 < a.M ? min(BN / 64, ceil_div(a.N - n0, 64)) : 0, first = out.half;
  const __nv_bfloat16* Dp = reinterpret_cast<const __nv_bfloat16*>(a.D);
  const __nv_bfloat16* D2p = reinterpret_cast<const __nv_bfloat16*>(a.D2);
  const bool diag = a.diag_add != 0.f && n0 < row0 + 32 && n0 + BN > row0;
  const long long goff = (long long)g * a.c_gstride;
  uint4 dpre[8];
  auto load_addend = [&](const __nv_bfloat16* P, int col) {      // 8 lanes per row: full 128-byte lines
#pragma unroll
    for (int i8 = 0; i8 < 8; ++i8) {
      const int grow = row0 + i8 * 4 + (lane >> 3);
      const int gcol = col + (lane & 7) * 8;
      dpre[i8] = (grow < a.M && gcol < a.N)
                     ? __ldg(reinterpret_cast<const uint4*>(P + goff + (long long)grow * a.ldd + gcol))
                     : make_uint4(0, 0, 0, 0);
    }
  };
  if (Dp != nullptr && first < slabs) load_addend(Dp, n0 + first * 64);          // under the wait for the accumulator
  if (!wait()) return false;
  if (first >= slabs) release();
  // the loop stays rolled: unrolled, the epilogue outgrows the instruction cache
#pragma unroll 1
  for (int sl = first; sl < slabs; sl += Stage::STEP) {
    const int col = n0 + sl * 64;
    uint32_t r[64];
    if (have_acc) {
      tmem_ld_32x32(t_row + sl * 64, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
      tmem_ld_32x32(t_row + sl * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int i = 0; i < 64; ++i) r[i] = 0u;
    }
    if (sl + Stage::STEP >= slabs) release();
#pragma unroll
    for (int i = 0; i < 64; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * scale);
    if (diag) {
#pragma unroll
      for (int i = 0; i < 64; ++i)
        if (col + i == row0 + lane) r[i] = __float_as_uint(__uint_as_float(r[i]) + a.diag_add);
    }
    uint8_t* sb = out_acquire(out, lane);
    if (Dp != nullptr) {
      // the addends pass through the staging buffer to reach the lane that owns their row
#pragma unroll 1
      for (int pass = 0; pass < (D2p != nullptr ? 2 : 1); ++pass) {
        const float bcoef = pass == 0 ? beta : beta2;
        if (pass == 1) load_addend(D2p, col);
#pragma unroll
        for (int i8 = 0; i8 < 8; ++i8) {
          const int rr = i8 * 4 + (lane >> 3);
          *reinterpret_cast<uint4*>(sb + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4)) = dpre[i8];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 q4 = *reinterpret_cast<const uint4*>(sb + lane * 128 + ((j ^ (lane & 7)) << 4));
          const __nv_bfloat162* pq = reinterpret_cast<const __nv_bfloat162*>(&q4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(pq[i]);
            r[j * 8 + 2 * i] = __float_as_uint(__uint_as_float(r[j * 8 + 2 * i]) + bcoef * f.x);
            r[j * 8 + 2 * i + 1] = __float_as_uint(__uint_as_float(r[j * 8 + 2 * i + 1]) + bcoef * f.y);
          }
        }
        __syncwarp();
      }
      if (sl + Stage::STEP < slabs) load_addend(Dp, col + 64 * Stage::STEP);
    }
    uint32_t p[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) p[i] = pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
    out_put_row(sb, lane, p);
    out_send(tmC, sb, lane, col, row0, g);
    if (mirror) {
      // two lanes hold a 2 x 2 block: they swap its off-diagonal corner and each writes one word of the transpose
      uint8_t* mb = out_acquire(out, lane);
      const bool odd = lane & 1;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const uint32_t give = odd ? (p[i] & 0xffffu) : (p[i] >> 16);
        const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 1);
        const uint32_t word = odd ? (got | (p[i] & 0xffff0000u)) : ((p[i] & 0xffffu) | (got << 16));
        *reinterpret_cast<uint32_t*>(mb + (2 * i + (odd ? 1 : 0)) * 64 + (lane >> 1) * 4) = word;
      }
      out_send(tmT, mb, lane, row0, col, g);
    }
  }
  return true;
}

// H = silu(gate) * up * scale, with the pre-activations G and U stored as well when asked for.  The accumulator holds
// HB gate columns followed by the HB up columns of the same outputs.
template <int HB, class Stage, class Release>
__device__ __forceinline__ void store_tile_swiglu(const GemmArgs& a, const CUtensorMap* tmH, const CUtensorMap* tmG,
                                                  const CUtensorMap* tmU, Stage& out, uint32_t t_row, bool have_acc,
                                                  int row0, int n0, int g, float scale, int lane, Release release) {
  const int slabs = row0 < a.M ? min(HB / 64, ceil_div(a.N - n0, 64)) : 0;
  if (out.half >= slabs) release();
  // Three results per slab, one after the other: reading tensor memory again costs less than holding both slabs in
  // registers (192 of them, which spilled).
#pragma unroll 1
  for (int sl = out.half; sl < slabs; sl += Stage::STEP) {
    const int col = n0 + sl * 64;
    const int last = a.U_out != nullptr ? 2 : (a.G_out != nullptr ? 1 : 0);
#pragma unroll 1
    for (int what = 0; what <= last; ++what) {
      if (what == 1 && a.G_out == nullptr) continue;
      uint32_t p[32];
      const uint32_t t_first = t_row + sl * 64 + (what == 2 ? HB : 0);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t x[32];
        if (have_acc) {
          tmem_ld_32x32(t_first + h * 32, x);
          if (what == 0) {
            uint32_t u[32];
            tmem_ld_32x32(t_row + HB + sl * 64 + h * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i)
              x[i] = __float_as_uint(silu_f(__uint_as_float(x[i])) * __uint_as_float(u[i]) * scale);
          } else {
            tmem_ld_wait();
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
          p[h * 16 + i] = pack_bf16(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1]));
      }
      if (sl + Stage::STEP >= slabs && what == last) release();
      uint8_t* sb = out_acquire(out, lane);
      out_put_row(sb, lane, p);
      out_send(what == 0 ? tmH : (what == 1 ? tmG : tmU), sb, lane, col, row0, g);
    }
  }
}

// MN-major tile of ROWS operand rows (memory [K][rows]) into shared memory as ROWS / 64 blocks of 64 k-rows x 128
// bytes.  A row count that is a multiple of 64 is described to TMA as (64, K, rows / 64) and the tile is one load;
// any other count (expert width 2464, vocabulary 50257) as (rows, K), where a load brings one block and the unit
// zero-fills what lies past the last row.  The second form costs ROWS / 64 issue slots of the producer thread
// instead of one, within the 0.4 us that a 256 x 256 x 64 step takes.
template <int ROWS>
__device__ __forceinline__ void load_mn_tile(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int k, int row, int g,
                                             int boxed) {
  if (!boxed) {
    tma_load_4d(dst, tm, bar, 0, k, row / 64, g);
  } else {
#pragma unroll
    for (int j = 0; j < ROWS / 64; ++j) tma_load_4d(dst + j * BK * 128, tm, bar, row + j * 64, k, 0, g);
  }
}
template <int ROWS>
__device__ __forceinline__ void load_mn_tile_pair(uint8_t* dst, const CUtensorMap* tm, uint32_t bar, int k, int row,
                                                  int g, int boxed) {
  if (!boxed) {
    tma_load_4d_pair(dst, tm, bar, 0, k, row / 64, g);
  } else {
#pragma unroll
    for (int j = 0; j < ROWS / 64; ++j) tma_load_4d_pair(dst + j * BK * 128, tm, bar, row + j * 64, k, 0, g);
  }
}

template <int BN, int A_MAJOR, int B_MAJOR>
__global__ void __launch_bounds__(threads_of(CTA_EPI_WARPS), 1)
umma_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmC,
                 const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, const GemmArgs args,
                 const int stages) {
  constexpr int B_STAGE_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN;  // two accumulators
  constexpr uint32_t IDESC = make_idesc_f16(BM, BN, /*bf16*/ 1, A_MAJOR, B_MAJOR);
  constexpr int MAX_STAGES = 8;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[MAX_STAGES];
  __shared__ uint64_t empty_bar[MAX_STAGES];
  __shared__ uint64_t tmem_full[2];
  __shared__ uint64_t tmem_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int2 ranges[RANGES_MAX];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], CTA_EPI_WARPS);  // one arrival per epilogue warp
    }
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_slot, TMEM_COLS);
    tmem_relinquish();
  }
  fill_ranges(args, ranges);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  const bool swiglu = args.epilogue == KMOE_EPI_SWIGLU;
  const int n_per_tile = swiglu ? BN / 2 : BN;  // output columns per tile
  int num_m = ceil_div(args.M, BM);
  if (args.mode == KMOE_GEMM_GROUPED_M) num_m = min(num_m, *args.num_m_tiles);
  const int num_n = ceil_div(args.N, n_per_tile);

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      Tile t;
      for (int idx = blockIdx.x; get_tile<BN>(args, idx, num_m, num_n, t, ranges); idx += gridDim.x) {
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!mbar_wait(&empty_bar[s], ph ^ 1)) {
            atomicExch(args.status, 1);
            goto teardown;
          }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE_BYTES;
          mbar_expect_tx(&full_bar[s], STAGE_BYTES);
          const int k = t.k0 + kb * BK;
          if (A_MAJOR == KMOE_MAJOR_K)
            tma_load_4d(sa, &tmA, &full_bar[s], k, t.m_tile * BM, 0, t.g_a);
          else
            load_mn_tile<BM>(sa, &tmA, &full_bar[s], k, t.m_tile * BM, t.g_a, args.a_boxed);
          if (!swiglu) {
            const bool second = args.k_split > 0 && k >= args.k_split;
            const CUtensorMap* tb = second ? &tmB2 : &tmB;
            const int kb2 = second ? k - args.k_split : k;
            if (B_MAJOR == KMOE_MAJOR_K)
              tma_load_4d(sb, tb, &full_bar[s], kb2, t.n_tile * BN, 0, t.g_b);
            else
              load_mn_tile<BN>(sb, tb, &full_bar[s], kb2, t.n_tile * BN, t.g_b, args.b_boxed);
          } else {
            constexpr int HB = BN / 2;
            if (B_MAJOR == KMOE_MAJOR_K) {
              tma_load_4d(sb, &tmB, &full_bar[s], k, t.n_tile * HB, 0, t.g_b);
              tma_load_4d(sb + B_STAGE_BYTES / 2, &tmB2, &full_bar[s], k, t.n_tile * HB, 0, t.g_b);
            } else {
              load_mn_tile<HB>(sb, &tmB, &full_bar[s], k, t.n_tile * HB, t.g_b, args.b_boxed);
              load_mn_tile<HB>(sb + B_STAGE_BYTES / 2, &tmB2, &full_bar[s], k, t.n_tile * HB, t.g_b, args.b_boxed);
            }
          }
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      Tile t;
      for (int idx = blockIdx.x; get_tile<BN>(args, idx, num_m, num_n, t, ranges); idx += gridDim.x) {
        const int acc = it & 1;
        const uint32_t acc_ph = (it >> 1) & 1;
        ++it;
        if (!mbar_wait(&tmem_empty[acc], acc_ph ^ 1)) {
          atomicExch(args.status, 2);
          goto teardown;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!mbar_wait(&full_bar[s], ph)) {
            atomicExch(args.status, 3);
            goto teardown;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_STAGE_BYTES;
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; ++k4) {
            // K-major: 16 bf16 = 32 B along the swizzled row. MN-major: 16 k-rows of 128 B.
            const uint32_t a_off = (A_MAJOR == KMOE_MAJOR_K) ? k4 * 32 : k4 * 16 * 128;
            const uint32_t b_off = (B_MAJOR == KMOE_MAJOR_K) ? k4 * 32 : k4 * 16 * 128;
            const uint64_t adesc = make_smem_desc_sw128(sa + a_off, (A_MAJOR == KMOE_MAJOR_K) ? 16 : BK * 128, 1024);
            const uint64_t bdesc = make_smem_desc_sw128(sb + b_off, (B_MAJOR == KMOE_MAJOR_K) ? 16 : BK * 128, 1024);
            umma_f16(d_tmem, adesc, bdesc, IDESC, (kb > 0 || k4 > 0) ? 1u : 0u);
          }
          umma_commit(&empty_bar[s]);  // frees the smem stage once these MMAs retire
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (t.k_blocks > 0)
          umma_commit(&tmem_full[acc]);
        else
          mbar_arrive(&tmem_full[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    int it = 0;
    Tile t;
    OutStage<CTA_EPI_WARPS> out(smem + stages * STAGE_BYTES, q);
    for (int idx = blockIdx.x; get_tile<BN>(args, idx, num_m, num_n, t, ranges); idx += gridDim.x) {
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      ++it;
      const bool have_acc = t.k_blocks > 0;
      const int row0 = t.m_tile * BM + q * 32;
      const int row = row0 + lane;
      const bool row_ok = row < args.M;
      float scale = args.alpha;
      float beta = args.beta;
      if (args.alpha_dev != nullptr) scale *= args.alpha_dev[t.g_c];
      if (args.beta_dev != nullptr) beta *= args.beta_dev[t.g_c];
      if (args.row_scale != nullptr && row_ok) scale *= args.row_scale[row];
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
      auto wait = [&]() {
        if (!mbar_wait(&tmem_full[acc], acc_ph)) {
          if (lane == 0) atomicExch(args.status, 4);
          return false;
        }
        tc_fence_after();
        return true;
      };
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[acc]);
      };
      if (!swiglu && !args.out_f32 && args.row_ptr == nullptr) {
        if (!store_tile_bf16<BN>(args, &tmC, &tmX, out, t_row, have_acc, row0, t.n_tile * BN, t.g_c, scale, beta, 0.f,
                                 false, lane, wait, release))
          goto teardown;
        continue;
      }
      if (!wait()) goto teardown;
      if (swiglu) {
        store_tile_swiglu<BN / 2>(args, &tmC, &tmX, &tmY, out, t_row, have_acc, row0, t.n_tile * (BN / 2), t.g_c, scale,
                                  lane, release);
        continue;
      }
      const long long coff = (long long)t.g_c * args.c_gstride + (long long)row * args.ldc;
      const long long doff = (long long)t.g_c * args.c_gstride + (long long)row * args.ldd;
      if (args.row_ptr != nullptr) {
        // Rows go to individual addresses, possibly on peer GPUs.  A lane holds one row, so a direct store
        // would emit 32 scattered 16-byte writes per instruction; the 64-column slab is staged in shared
        // memory instead and written back with 8 lanes per row: four full 128-byte lines per instruction.
        const long long row_addr = row_ok ? args.row_ptr[row] : 0;
        __nv_bfloat16(*stg)[72] = reinterpret_cast<__nv_bfloat16(*)[72]>(out.base);      // 32 rows, within 8 KB
        const __nv_bfloat16* Dp = reinterpret_cast<const __nv_bfloat16*>(args.D);
#pragma unroll 1
        for (int c = 0; c < BN; c += 64) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            if (have_acc) {
              tmem_ld_32x32(t_row + c + h * 32, r);
              tmem_ld_wait();
            }
            const int col = t.n_tile * BN + c + h * 32;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = have_acc ? __uint_as_float(r[j + i]) * scale : 0.f;
              if (Dp != nullptr && row_ok && col + j < args.N) {
                float d[8];
                load8(Dp + doff + col + j, d);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] += beta * d[i];
              }
              store8<__nv_bfloat16>(&stg[lane][h * 32 + j], v);
            }
          }
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int rr = it * 4 + (lane >> 3);
            const int cc = (lane & 7) * 8;
            const long long addr = __shfl_sync(0xffffffffu, row_addr, rr);
            const int gcol = t.n_tile * BN + c + cc;
            if (addr != 0 && gcol < args.N)
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(addr) + gcol) =
                  *reinterpret_cast<const uint4*>(&stg[rr][cc]);
          }
          __syncwarp();
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          if (have_acc) {
            tmem_ld_32x32(t_row + c, r);
            tmem_ld_wait();
          }
          const int col = t.n_tile * BN + c;
          if (row_ok && col < args.N) epilogue_store_chunk_f32(args, r, have_acc, coff, doff, col, scale, beta);
        }
      }
      release();
    }
  }

teardown:
  if (warp >= 2 && lane == 0) tma_store_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------ CTA-pair kernel
// The same GEMM with tcgen05.mma.cta_group::2: the two CTAs of a cluster share one 256 x BN tile.  Each CTA
// loads its own 128 rows of A and its own half of B's columns (plain per-CTA TMA loads), the even CTA issues
// 256 x BN x 16 MMAs that read both CTAs' shared memory, and each CTA ends up with its 128 rows of the
// accumulator in its own tensor memory.  Halving the B traffic per CTA is what lifts the tensor pipe off the
// shared-memory bandwidth limit of the single-CTA 128 x 256 tile.
//
// Barriers: `full` lives in the leader and is credited by both CTAs' loads; `empty` and `tmem_full` exist in
// both CTAs and are signalled by the leader's commits (multicast arrive); `tmem_empty` lives in the leader
// and collects the epilogue warps of both CTAs.  All schedules, all epilogues except per-row destination addresses.
constexpr int PAIR_TM = 2 * BM;
// Expert-padded schedule: blocks per expert (counting the padding) from which pairs are taken.  Up / down / dH products
// in µs, pairs against single CTAs, at d = 2048, f = 2816: 2.6 live blocks per expert 459/234/235 against 434/219/226,
// 4.6 blocks 351/180/178 against 343/175/185, 6.4 blocks 309/157/156 against 310/165/167, 12.4 blocks 268/132/135 against
// 272/141/149.
constexpr int GROUPED_PAIR_MIN = 7;

// Eight epilogue warps instead of four, by the reduction of a tile (the mean one of ragged products).  They finish a tile
// sooner, which counts while the epilogue is longer than the reduction it runs beside; where it is not, twice as many
// warps only take shared memory and issue slots from the products.  The more an epilogue does per tile, the longer the
// reduction up to which it counts.  In us, eight against four:
//   plain bf16, more tiles than pairs: 16 products of 2048 x 2816 over K = 128 52 / 60, 256 57 / 64, 384 69 / 72, 448 76 / 75,
//     768 115 / 111, 1536 200 / 197; 64 of 1792 x 2464 over 128 143 / 172, 384 218 / 220, 448 248 / 231;
//     8192 x 4096 over 128 22.7 / 24.8, 384 28.3 / 29.0, 640 36.0 / 34.7.  One round of tiles: 0.2 to 0.6 us more.
//     Uneven groups, whose short ones gain what the long ones lose: as 1 / rank over 16 groups, mean 768, 143 / 142; even 116 / 112.
//   SwiGLU with both pre-activations: 4096 x 2048 over 512 27.1 / 30.9, 4096 x 4096 over 1536 76.9 / 74.8.
//   an addend: 8192 x 4096 over 512 57 / 79, 1024 60 / 80, 1536 77 / 82, 2048 97 / 98, 4096 185 / 183, 8192 380 / 366.
//   fp32 results: never, 2048 x 2048 over 256 15.5 / 12.4, 8192 x 4096 over 1024 80 / 76.
constexpr int WIDE_K_PLAIN = 384, WIDE_K_SWIGLU = 512, WIDE_K_ADDEND = 2048;

template <int BN, int A_MAJOR, int B_MAJOR, int EPI_WARPS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads_of(EPI_WARPS), 1)
umma_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmC,
                 const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY, const GemmArgs args,
                 const int stages) {
  constexpr int HALF_N = BN / 2;
  constexpr int B_STAGE_BYTES = HALF_N * BK * 2;
  constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;   // per CTA
  constexpr uint32_t TMEM_COLS = 2 * BN;
  constexpr uint32_t IDESC = make_idesc_f16(PAIR_TM, BN, /*bf16*/ 1, A_MAJOR, B_MAJOR);
  constexpr int MAX_STAGES = 8;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[MAX_STAGES];
  __shared__ uint64_t empty_bar[MAX_STAGES];
  __shared__ uint64_t tmem_full[2];
  __shared__ uint64_t tmem_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ __align__(8) uint16_t pair_list[PAIR_LIST_MAX];
  int2* ranges = reinterpret_cast<int2*>(pair_list);      // one schedule has the list, another the ranges
  static_assert(sizeof(pair_list) >= RANGES_MAX * sizeof(int2), "ranges fit");
  __shared__ int pair_list_len;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 2 * EPI_WARPS);   // the epilogue warps of both CTAs
    }
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {                    // collective over the pair: the same warp of both CTAs
    tmem_alloc_pair(&tmem_base_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  if (warp == 2 && args.mode == KMOE_GEMM_GROUPED_M) {
    const int n = build_pair_list(args.tile_group, min(ceil_div(args.M, BM), *args.num_m_tiles), pair_list, lane);
    if (lane == 0) pair_list_len = n;
  }
  fill_ranges(args, ranges);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                 // the peer's barriers exist before anything is signalled across
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  const bool swiglu = args.epilogue == KMOE_EPI_SWIGLU;
  const int n_per_tile = swiglu ? BN / 2 : BN;
  const int num_m = args.mode == KMOE_GEMM_GROUPED_M ? pair_list_len : ceil_div(args.M, PAIR_TM);
  const int num_n = ceil_div(args.N, n_per_tile);

  auto leave = [&]() {                // every wait before it is bounded, so all warps come
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();               // nothing of the peer may still point at this CTA's memory
  };

  constexpr bool wide = EPI_WARPS == 8;
  constexpr int FIRST_EPI = wide ? 4 : 2;
  if (warp < FIRST_EPI) {
    if (wide) set_regs_down<ROLE_REGS>();
    {
  if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs)
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      Tile t;
      for (int idx = pair; get_tile<BN, PAIR_TM>(args, idx, num_m, num_n, t, ranges, pair_list); idx += num_pairs) {
        const int arow = t.row + (int)rank * BM;
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!mbar_wait(&empty_bar[s], ph ^ 1)) {
            atomicExch(args.status, 11);
            goto role_done;
          }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE_BYTES;
          if (leader) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
          const uint32_t fb = map_to_cta(&full_bar[s], 0);
          const int k = t.k0 + kb * BK;
          if (A_MAJOR == KMOE_MAJOR_K)
            tma_load_4d_pair(sa, &tmA, fb, k, arow, 0, t.g_a);
          else
            load_mn_tile_pair<BM>(sa, &tmA, fb, k, arow, t.g_a, args.a_boxed);
          // B: this CTA's half of the tile's columns; with the SwiGLU epilogue the halves are the gate
          // weight (leader) and the up weight (peer), so accumulator columns [0, BN/2) hold the gate
          const bool second = !swiglu && args.k_split > 0 && k >= args.k_split;
          const CUtensorMap* tb = ((swiglu && !leader) || second) ? &tmB2 : &tmB;
          const int kb2 = second ? k - args.k_split : k;
          const int brow = swiglu ? t.n_tile * HALF_N : t.n_tile * BN + (int)rank * HALF_N;
          if (B_MAJOR == KMOE_MAJOR_K)
            tma_load_4d_pair(sb, tb, fb, kb2, brow, 0, t.g_b);
          else
            load_mn_tile_pair<HALF_N>(sb, tb, fb, kb2, brow, t.g_b, args.b_boxed);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer (leader only)
    if (leader && elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      Tile t;
      for (int idx = pair; get_tile<BN, PAIR_TM>(args, idx, num_m, num_n, t, ranges, pair_list); idx += num_pairs) {
        const int acc = it & 1;
        const uint32_t acc_ph = (it >> 1) & 1;
        ++it;
        if (!mbar_wait(&tmem_empty[acc], acc_ph ^ 1)) {
          atomicExch(args.status, 12);
          goto role_done;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < t.k_blocks; ++kb) {
          if (!mbar_wait(&full_bar[s], ph)) {
            atomicExch(args.status, 13);
            goto role_done;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_STAGE_BYTES;
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; ++k4) {
            const uint32_t a_off = (A_MAJOR == KMOE_MAJOR_K) ? k4 * 32 : k4 * 16 * 128;
            const uint32_t b_off = (B_MAJOR == KMOE_MAJOR_K) ? k4 * 32 : k4 * 16 * 128;
            const uint64_t adesc = make_smem_desc_sw128(sa + a_off, (A_MAJOR == KMOE_MAJOR_K) ? 16 : BK * 128, 1024);
            const uint64_t bdesc = make_smem_desc_sw128(sb + b_off, (B_MAJOR == KMOE_MAJOR_K) ? 16 : BK * 128, 1024);
            umma_f16_pair(d_tmem, adesc, bdesc, IDESC, (kb > 0 || k4 > 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[s], 3);      // frees the stage in both CTAs
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (t.k_blocks > 0) {
          umma_commit_pair(&tmem_full[acc], 3);
        } else {
          mbar_arrive(&tmem_full[acc]);
          mbar_arrive_cluster_relaxed(map_to_cta(&tmem_full[acc], 1));
        }
      }
    }
  }
    }
  role_done:
    __syncwarp();
    leave();
    if (warp == 1) {
      tc_fence_after();
      tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
  } else {
    if (wide) set_regs_up<EPI_REGS>();
    {
    // ------------------------------------------------------------ epilogue (both CTAs)
    const int q = warp & 3;
    int it = 0;
    Tile t;
    OutStage<EPI_WARPS> out(smem + stages * STAGE_BYTES, warp - FIRST_EPI);
    for (int idx = pair; get_tile<BN, PAIR_TM>(args, idx, num_m, num_n, t, ranges, pair_list); idx += num_pairs) {
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      ++it;
      const bool have_acc = t.k_blocks > 0;
      // rows of another expert: past the end, so that nothing is stored
      const int row0 = leader || t.rows_ok ? t.row + (int)rank * BM + q * 32 : args.M;
      const int row = row0 + lane;
      const bool row_ok = row < args.M;
      float scale = args.alpha;
      float beta = args.beta, beta2 = args.beta2;
      if (args.alpha_dev != nullptr) scale *= args.alpha_dev[t.g_c];
      if (args.beta_dev != nullptr) {
        beta *= args.beta_dev[t.g_c];
        beta2 *= args.beta_dev[t.g_c];
      }
      if (args.row_scale != nullptr && row_ok) scale *= args.row_scale[row];
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
      auto wait = [&]() {
        if (!mbar_wait(&tmem_full[acc], acc_ph)) {
          if (lane == 0) atomicExch(args.status, 14);
          return false;
        }
        tc_fence_after();
        return true;
      };
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (leader) mbar_arrive(&tmem_empty[acc]);
          else mbar_arrive_cluster_relaxed(map_to_cta(&tmem_empty[acc], 0));
        }
      };
      if (!swiglu && !args.out_f32) {
        // symmetric product: a tile strictly above the diagonal also writes its transpose
        const bool mirror = args.sym_upper && t.n_tile * BN >= (t.m_tile + 1) * PAIR_TM;
        if (!store_tile_bf16<BN>(args, &tmC, &tmX, out, t_row, have_acc, row0, t.n_tile * BN, t.g_c, scale, beta, beta2,
                                 mirror, lane, wait, release))
          goto epi_done;
        continue;
      }
      if (!wait()) goto epi_done;
      if (swiglu) {
        store_tile_swiglu<HALF_N>(args, &tmC, &tmX, &tmY, out, t_row, have_acc, row0, t.n_tile * HALF_N, t.g_c, scale,
                                  lane, release);
        continue;
      }
      const long long goff = (long long)t.g_c * args.c_gstride;
      const long long coff = goff + (long long)row * args.ldc;
      const long long doff = goff + (long long)row * args.ldd;
#pragma unroll 1
      for (int c = wide ? out.half * (BN / 2) : 0; c < (wide ? (out.half + 1) * (BN / 2) : BN); c += 32) {
        uint32_t r[32];
        if (have_acc) {
          tmem_ld_32x32(t_row + c, r);
          tmem_ld_wait();
        }
        const int col = t.n_tile * BN + c;
        if (row_ok && col < args.N) epilogue_store_chunk_f32(args, r, have_acc, coff, doff, col, scale, beta);
      }
      release();
    }
    }
  epi_done:
    if (lane == 0) tma_store_wait_all();
    __syncwarp();
    leave();
  }
}

// Fills the tiles that a symmetric GEMM skipped: C[g][i][j] = C[g][j][i] for every 32x32 block that lies in a
// tile entirely below the diagonal.  grid = (n/32, n/32, groups), block = (32, 8).
__global__ void sym_mirror_kernel(__nv_bfloat16* __restrict__ C, int n, long long ldc, long long gstride, int bn,
                                  int tm) {
  const int bx = blockIdx.x, by = blockIdx.y;
  const int mt = (by * 32) / tm, nt = (bx * 32) / bn;
  if ((nt + 1) * bn > mt * tm) return;                      // destination was computed
  __shared__ __nv_bfloat16 tile[32][33];
  __nv_bfloat16* Cg = C + (long long)blockIdx.z * gstride;
  for (int r = threadIdx.y; r < 32; r += 8)                  // source block: rows 32*bx.., cols 32*by..
    tile[r][threadIdx.x] = Cg[(long long)(bx * 32 + r) * ldc + by * 32 + threadIdx.x];
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8)
    Cg[(long long)(by * 32 + r) * ldc + bx * 32 + threadIdx.x] = tile[threadIdx.x][r];
}

// ------------------------------------------------------------------ host side
using TmapKey = std::tuple<const void*, int, long long, long long, long long, long long, int, int>;
static std::map<TmapKey, CUtensorMap> g_tmap_cache;
static std::mutex g_tmap_mutex;

// Operand tensor map (bf16, 128B swizzle), always rank 4 so one TMA instruction form serves all cases.
//   K-major : dims {K, rows, 1, G}       box {64, tile_rows, 1, 1}
//   MN-major: dims {64, K, rows/64, G}   box {64, 64, tile_rows/64, 1}   (memory is [K][rows], rows contiguous)
//             dims {rows, K, 1, G}       box {64, 64, 1, 1}              when rows % 64 != 0 (see load_mn_tile)
static int make_operand_tmap(CUtensorMap* out, const void* base, int major, long long rows, long long K,
                             long long ld, long long gstride, int groups, int tile_rows) {
  TmapKey key{base, major, rows, K, ld, gstride, groups, tile_rows};
  {
    std::lock_guard<std::mutex> lk(g_tmap_mutex);
    auto it = g_tmap_cache.find(key);
    if (it != g_tmap_cache.end()) {
      *out = it->second;
      return 0;
    }
  }
  cuuint64_t dims[4];
  cuuint64_t strides[3];
  cuuint32_t box[4];
  const long long gs = (groups > 1 && gstride > 0) ? gstride : (major == KMOE_MAJOR_K ? rows * ld : K * ld);
  const int G = (groups > 1 && gstride > 0) ? groups : 1;
  if (major == KMOE_MAJOR_K) {
    dims[0] = (cuuint64_t)K; dims[1] = (cuuint64_t)rows; dims[2] = 1; dims[3] = (cuuint64_t)G;
    strides[0] = (cuuint64_t)ld * 2; strides[1] = (cuuint64_t)rows * ld * 2; strides[2] = (cuuint64_t)gs * 2;
    box[0] = BK; box[1] = (cuuint32_t)tile_rows; box[2] = 1; box[3] = 1;
  } else {
    if (rows % 64 != 0) {
      dims[0] = (cuuint64_t)rows; dims[1] = (cuuint64_t)K; dims[2] = 1; dims[3] = (cuuint64_t)G;
      strides[0] = (cuuint64_t)ld * 2; strides[1] = (cuuint64_t)K * ld * 2; strides[2] = (cuuint64_t)gs * 2;
      box[0] = 64; box[1] = BK; box[2] = 1; box[3] = 1;
    } else {
    dims[0] = 64; dims[1] = (cuuint64_t)K; dims[2] = (cuuint64_t)(rows / 64); dims[3] = (cuuint64_t)G;
    strides[0] = (cuuint64_t)ld * 2; strides[1] = 128; strides[2] = (cuuint64_t)gs * 2;
    box[0] = 64; box[1] = BK; box[2] = (cuuint32_t)(tile_rows / 64); box[3] = 1;
    }
  }
  const int rc = encode_bf16_4d(out, base, dims, strides, box);
  if (rc) return rc;
  {
    std::lock_guard<std::mutex> lk(g_tmap_mutex);
    if (g_tmap_cache.size() > 4096) g_tmap_cache.clear();
    g_tmap_cache[key] = *out;
  }
  return 0;
}

// Output tensor map (bf16): dims {N, rows, 1, G}.  Plain: box {64, 32}, 128B swizzle, the staging buffer of an epilogue
// warp.  Transposed tiles of a symmetric product: box {32, 64} without swizzle.
static int make_output_tmap(CUtensorMap* out, const void* base, long long rows, long long N, long long ld,
                            long long gstride, int groups, bool transposed) {
  TmapKey key{base, transposed ? 3 : 2, rows, N, ld, gstride, groups, 0};
  {
    std::lock_guard<std::mutex> lk(g_tmap_mutex);
    auto it = g_tmap_cache.find(key);
    if (it != g_tmap_cache.end()) {
      *out = it->second;
      return 0;
    }
  }
  const long long gs = groups > 1 ? gstride : rows * ld;
  const cuuint64_t dims[4] = {(cuuint64_t)N, (cuuint64_t)rows, 1, (cuuint64_t)groups};
  const cuuint64_t strides[3] = {(cuuint64_t)ld * 2, (cuuint64_t)rows * ld * 2, (cuuint64_t)gs * 2};
  const cuuint32_t box[4] = {transposed ? 32u : 64u, transposed ? 64u : 32u, 1, 1};
  const int rc = encode_bf16_4d(out, base, dims, strides, box,
                                transposed ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  {
    std::lock_guard<std::mutex> lk(g_tmap_mutex);
    if (g_tmap_cache.size() > 4096) g_tmap_cache.clear();
    g_tmap_cache[key] = *out;
  }
  return 0;
}

template <int BN, int AM, int BMj>
static int launch_variant(const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tB2, const CUtensorMap& tC,
                          const CUtensorMap& tX, const CUtensorMap& tY, const GemmArgs& args, int grid,
                          cudaStream_t stream) {
  constexpr int stage_bytes = A_STAGE_BYTES + BN * BK * 2;
  int stages = (192 * 1024) / stage_bytes;      // operand ring beside the 32 KB of output staging
  if (stages > 8) stages = 8;
  const int smem = stages * stage_bytes + OUT_STAGE_BYTES + 1024;
  auto kern = umma_gemm_kernel<BN, AM, BMj>;
  static SmemLimit limit;
  if (!limit.raise(kern, smem)) return -20;
  kern<<<grid, threads_of(CTA_EPI_WARPS), smem, stream>>>(tA, tB, tB2, tC, tX, tY, args, stages);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

template <int BN, int AM, int BMj, int EPI_WARPS>
static int launch_pair_variant(const CUtensorMap& tA, const CUtensorMap& tB, const CUtensorMap& tB2,
                               const CUtensorMap& tC, const CUtensorMap& tX, const CUtensorMap& tY,
                               const GemmArgs& args, long long pair_tiles, int sms, cudaStream_t stream) {
  constexpr int stage_bytes = A_STAGE_BYTES + (BN / 2) * BK * 2;
  int stages = (192 * 1024) / stage_bytes;
  if (stages > 8) stages = 8;
  const int smem = stages * stage_bytes + OUT_STAGE_BYTES + 1024;
  auto kern = umma_gemm_pair_kernel<BN, AM, BMj, EPI_WARPS>;
  static SmemLimit limit;
  if (!limit.raise(kern, smem)) return -20;
  static int max_clusters = 0;
  if (max_clusters == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * (sms / 2)));
    cfg.blockDim = dim3(threads_of(EPI_WARPS));
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) n = sms / 2;
    max_clusters = n;
  }
  long long pairs = pair_tiles < max_clusters ? pair_tiles : max_clusters;
  if (pairs < 1) pairs = 1;
  kern<<<(unsigned)(2 * pairs), threads_of(EPI_WARPS), smem, stream>>>(tA, tB, tB2, tC, tX, tY, args, stages);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

// KMOE_GEMM_PAIR=0 keeps every GEMM on the single-CTA kernel.
static bool pair_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("KMOE_GEMM_PAIR");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

}  // namespace kmoe

extern "C" void kmoe_gemm_clear_tensormap_cache(void) {
  std::lock_guard<std::mutex> lk(kmoe::g_tmap_mutex);
  kmoe::g_tmap_cache.clear();
}

extern "C" int kmoe_gemm(const KmoeGemmDesc* d, cudaStream_t stream) {
  using namespace kmoe;
  // 16-byte output vectors; the pitches of the operands are checked where their tensor maps are made (the lengths
  // themselves are free: TMA zero-fills past the end of a row and past the last row)
  if (d->N % 8 != 0 || d->ldc % (d->out_f32 ? 4 : 8) != 0) return -1;
  if (d->b_rows < 0 || d->b_rows > d->N || d->b_klen < 0 || d->b_klen > (d->k_split ? d->k_split : d->K)) return -7;
  if (d->K <= 0 || d->M <= 0 || d->N <= 0) return -2;
  if (d->c_row_ptr != nullptr && (d->out_f32 || d->epilogue != KMOE_EPI_STORE)) return -3;
  if (d->k_split != 0 && (d->k_split % BK || d->k_split <= 0 || d->k_split >= d->K || d->B2 == nullptr ||
                          d->epilogue != KMOE_EPI_STORE || d->k_begin != nullptr))
    return -5;
  const bool swiglu = d->epilogue == KMOE_EPI_SWIGLU;
  // narrow outputs use the 128-wide tile so more CTAs get work
  const int n_tiles_256 = (d->N + (swiglu ? 127 : 255)) / (swiglu ? 128 : 256);
  const long long m_tiles = (d->M + BM - 1) / BM;
  const long long groups = d->mode == KMOE_GEMM_BATCHED ? d->groups : 1;
  int sms = d->num_sms;
  if (sms <= 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  // CTA-pair kernel (256-row tiles): everything except per-row destination addresses.  On the expert-padded schedule
  // (128-row blocks) an expert with an odd number of blocks wastes half a tile, at most `groups` blocks in all, so the
  // pair is taken from GROUPED_PAIR_MIN blocks per expert up.
  const bool grouped_pair = d->mode == KMOE_GEMM_GROUPED_M && m_tiles <= PAIR_LIST_MAX &&
                            m_tiles >= (long long)GROUPED_PAIR_MIN * d->groups;
  const bool pair = pair_enabled() && (d->mode != KMOE_GEMM_GROUPED_M || grouped_pair) && d->c_row_ptr == nullptr &&
                    d->M > BM;
  const int TM = pair ? PAIR_TM : BM;
  const long long tm_tiles = pair && grouped_pair ? (m_tiles + d->groups) / 2 : (d->M + TM - 1) / TM;
  const int units = pair ? sms / 2 : sms;       // CTAs or CTA pairs that run at once
  // 256-wide tiles unless that would leave most of the machine idle.  A CTA pair on 256 x 128 tiles asks the L2
  // for about 1.5x the bytes per FLOP of a 256 x 256 tile and runs at nearly the same time per reduction block,
  // so two waves of narrow tiles are slower than one partly filled wave of wide ones.
  const long long tiles256 = tm_tiles * n_tiles_256 * groups;
  const bool use256 = swiglu || (d->N >= 256 && (pair ? 2 * tiles256 > units : tiles256 >= units));
  const int BN = use256 ? 256 : 128;
  const int b_box_rows = pair ? BN / 2 : (swiglu ? BN / 2 : BN);

  GemmArgs a;
  a.C = d->C; a.D = d->D; a.D2 = d->D2; a.beta2 = d->beta2; a.G_out = d->G_out; a.U_out = d->U_out;
  a.mode = d->mode; a.epilogue = d->epilogue;
  a.M = d->M; a.N = d->N; a.K = d->K; a.groups = d->groups;
  a.ldc = d->ldc; a.ldd = d->ldd ? d->ldd : d->ldc; a.c_gstride = d->c_gstride;
  a.a_grouped = d->a_gstride != 0; a.b_grouped = d->b_gstride != 0;
  a.tile_group = d->tile_group; a.num_m_tiles = d->num_m_tiles;
  a.k_begin = d->k_begin; a.k_len = d->k_len;
  a.out_f32 = d->out_f32; a.alpha = d->alpha; a.beta = d->beta;
  a.row_scale = d->row_scale; a.row_ptr = d->c_row_ptr; a.status = d->status;
  a.alpha_dev = d->alpha_dev; a.beta_dev = d->beta_dev;
  a.sym_upper = d->sym_upper;
  a.diag_add = d->diag_add;
  a.k_split = d->k_split;
  if (d->sym_upper && (d->M != d->N || swiglu || d->mode == KMOE_GEMM_GROUPED_M || d->out_f32 || d->N % 32 ||
                       (d->D != nullptr && !pair)))
    return -4;
  // the second addend exists in the bf16 epilogue of the CTA-pair kernel only
  if (d->D2 != nullptr && (!pair || swiglu || d->out_f32 || d->D == nullptr)) return -6;

  // The reduction extent seen by TMA: ragged batched GEMMs index a shared [sum K, rows] buffer.
  long long k_extent_a = d->K, k_extent_b = d->K;
  if (d->mode == KMOE_GEMM_BATCHED && d->k_begin != nullptr) {
    k_extent_a = d->a_gstride == 0 ? (long long)d->K : d->K;
    k_extent_b = k_extent_a;
  }
  const int a_groups = (d->mode == KMOE_GEMM_BATCHED && d->a_gstride != 0) ? d->groups : 1;
  const int b_groups = d->b_gstride != 0 ? d->groups : 1;
  const int n_rows = d->b_rows > 0 ? d->b_rows : d->N;
  a.a_boxed = d->a_major == KMOE_MAJOR_MN && d->M % 64 != 0;
  a.b_boxed = d->b_major == KMOE_MAJOR_MN && n_rows % 64 != 0;
  CUtensorMap tA, tB, tB2;
  int rc = make_operand_tmap(&tA, d->A, d->a_major, d->M, k_extent_a, d->lda, d->a_gstride, a_groups, BM);
  if (rc) return rc;
  if (d->k_split > 0) k_extent_b = d->k_split;
  if (d->b_klen > 0) k_extent_b = d->b_klen;
  rc = make_operand_tmap(&tB, d->B, d->b_major, n_rows, k_extent_b, d->ldb, d->b_gstride, b_groups, b_box_rows);
  if (rc) return rc;
  if (d->k_split > 0) {
    rc = make_operand_tmap(&tB2, d->B2, d->b_major, n_rows, d->b_klen > 0 ? d->b_klen : d->K - d->k_split, d->ldb,
                           d->b_gstride, b_groups, b_box_rows);
    if (rc) return rc;
  } else if (swiglu) {
    rc = make_operand_tmap(&tB2, d->B2, d->b_major, n_rows, k_extent_b, d->ldb, d->b_gstride, b_groups, b_box_rows);
    if (rc) return rc;
  } else {
    tB2 = tB;
  }
  // outputs that leave by TMA stores: everything but fp32 results and per-row destinations
  CUtensorMap tC = tA, tX = tA, tY = tA;
  if (!d->out_f32 && d->c_row_ptr == nullptr) {
    const int c_groups = (int)groups;
    rc = make_output_tmap(&tC, d->C, d->M, d->N, d->ldc, d->c_gstride, c_groups, false);
    if (!rc && swiglu && d->G_out) rc = make_output_tmap(&tX, d->G_out, d->M, d->N, d->ldc, d->c_gstride, c_groups, false);
    if (!rc && swiglu && d->U_out) rc = make_output_tmap(&tY, d->U_out, d->M, d->N, d->ldc, d->c_gstride, c_groups, false);
    if (!rc && d->sym_upper && pair) rc = make_output_tmap(&tX, d->C, d->M, d->N, d->ldc, d->c_gstride, c_groups, true);
    if (rc) return rc;
  }
  const int n_per_tile = swiglu ? BN / 2 : BN;
  long long total = tm_tiles * ((d->N + n_per_tile - 1) / n_per_tile) * groups;
  if (d->sym_upper) {
    const long long nn = (d->N + BN - 1) / BN;
    long long kept = 0;
    for (long long m = 0; m < tm_tiles; ++m) kept += nn - std::min<long long>(nn, (m * TM) / BN);
    total = kept * groups;
  }
  int grid = (int)(total < sms ? total : sms);
  if (grid < 1) grid = 1;

  const long long mean_k = (long long)d->K / (d->k_begin != nullptr && d->groups > 1 ? d->groups : 1);
  const bool wide = !d->out_f32 && (d->D != nullptr ? mean_k <= WIDE_K_ADDEND
                                    : swiglu        ? mean_k <= WIDE_K_SWIGLU
                                                    : mean_k <= WIDE_K_PLAIN && total > units);
  int lrc = 0;
#define KMOE_LAUNCH_PAIR(BN_, AM_, BM_)                                                                        \
  lrc = wide ? launch_pair_variant<BN_, AM_, BM_, 8>(tA, tB, tB2, tC, tX, tY, a, total, sms, stream)           \
             : launch_pair_variant<BN_, AM_, BM_, 4>(tA, tB, tB2, tC, tX, tY, a, total, sms, stream)
#define KMOE_LAUNCH(BN_, AM_, BM_) lrc = launch_variant<BN_, AM_, BM_>(tA, tB, tB2, tC, tX, tY, a, grid, stream)
  if (pair && BN == 256) {
    if (d->a_major == 0 && d->b_major == 0) KMOE_LAUNCH_PAIR(256, 0, 0);
    else if (d->a_major == 0 && d->b_major == 1) KMOE_LAUNCH_PAIR(256, 0, 1);
    else if (d->a_major == 1 && d->b_major == 0) KMOE_LAUNCH_PAIR(256, 1, 0);
    else KMOE_LAUNCH_PAIR(256, 1, 1);
  } else if (pair) {
    if (d->a_major == 0 && d->b_major == 0) KMOE_LAUNCH_PAIR(128, 0, 0);
    else if (d->a_major == 0 && d->b_major == 1) KMOE_LAUNCH_PAIR(128, 0, 1);
    else if (d->a_major == 1 && d->b_major == 0) KMOE_LAUNCH_PAIR(128, 1, 0);
    else KMOE_LAUNCH_PAIR(128, 1, 1);
  } else if (BN == 256) {
    if (d->a_major == 0 && d->b_major == 0) KMOE_LAUNCH(256, 0, 0);
    else if (d->a_major == 0 && d->b_major == 1) KMOE_LAUNCH(256, 0, 1);
    else if (d->a_major == 1 && d->b_major == 0) KMOE_LAUNCH(256, 1, 0);
    else KMOE_LAUNCH(256, 1, 1);
  } else {
    if (d->a_major == 0 && d->b_major == 0) KMOE_LAUNCH(128, 0, 0);
    else if (d->a_major == 0 && d->b_major == 1) KMOE_LAUNCH(128, 0, 1);
    else if (d->a_major == 1 && d->b_major == 0) KMOE_LAUNCH(128, 1, 0);
    else KMOE_LAUNCH(128, 1, 1);
  }
#undef KMOE_LAUNCH
#undef KMOE_LAUNCH_PAIR
  if (lrc) return lrc;
  if (d->sym_upper && !pair) {
    // the tiles below the diagonal were skipped: mirror them from the computed upper part (the CTA-pair
    // kernel writes the transposed tiles from its epilogue instead)
    dim3 mg((unsigned)(d->N / 32), (unsigned)(d->N / 32), (unsigned)groups);
    sym_mirror_kernel<<<mg, dim3(32, 8), 0, stream>>>((__nv_bfloat16*)d->C, d->N, d->ldc, d->c_gstride, BN, TM);
    if (cudaGetLastError() != cudaSuccess) return -22;
  }
  return 0;
}
