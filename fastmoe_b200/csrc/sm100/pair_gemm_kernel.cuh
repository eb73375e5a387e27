// Grouped GEMM on CTA pairs (tcgen05 cta_group::2) with 256 x 256 tiles: weight gradients, and input
// gradients of many rows that apply an activation's derivative (the other row modes without an
// exchange: slim_gemm_kernel.cuh).
//
// A pair of CTAs (one cluster, two neighbouring SMs) works on a 256 x 256 output tile: CTA r
// holds rows [128 r, 128 r + 128) of A, columns [128 r, 128 r + 128) of B and the accumulators of
// its rows.  Per 64-wide K block an SM loads 32 KB where a 128 x 256 tile on one SM loads 48 KB.
// Measured, bf16, 8192 rows, 2 experts, 1024 <-> 4096: input gradient with GELU's derivative 67.3 us,
// weight gradient with the bias gradient 57.1 us (1200 TFLOP/s), where the single-CTA kernel took 78.4 and 70.1
// us.  What bounds it: the last of the waves (128 tiles on 74 pairs), the L2 (8 TB/s to the SMs at 0.6 us per K
// block) and, with an activation, the epilogue.
//
// Roles of a CTA (384 threads), persistent over the tiles of its pair:
//   warp 0      TMA producer, one lane: this CTA's halves of A and B into a 5-stage ring; the
//               bytes of both CTAs are counted on CTA 0's barrier of the stage;
//   warp 1      CTA 0: one lane issues the pair's MMAs and commits to both CTAs' barriers; in
//               both CTAs the warp owns the TMEM allocation;
//   warp 2      weight gradient: an expert's last rows, where they do not fill an MMA step of 16, by plain
//               loads into a buffer of their own, filled up with zeros, a tile or two ahead;
//   warp 3      weight gradient: zeroes the gradients of experts without rows, beside the MMAs;
//   warps 4-11  epilogue: as in the single-CTA kernel, 32 rows x 128 columns per warp; whole rows of
//               32 leave by TMA.
// The ring brings whole K blocks, of which the MMA steps that are full of the expert's rows are issued.
// The step that is not has its operands beside the ring: zeroed in the ring after they had landed, the rows
// past the end held every tile of a ragged expert up by 1.3 us (16 experts, 1024 <-> 4096: 375 rows each
// 70.2 us against 51.9 with 384; now 52.8).
#pragma once
#include "grouped_gemm_kernel.cuh"
#include "launch.cuh"

namespace fmoe {
namespace pg {

using gg::Cvt;
using gg::Packed32;

constexpr int CTA_M = 128;                  // rows of A and of the output per CTA
constexpr int TILE_M = 2 * CTA_M;
constexpr int TILE_N = 256;
constexpr int CTA_N = TILE_N / 2;           // columns of B per CTA
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int STAGES = 5;
constexpr int BOX_BYTES = 64 * BK * 2;      // one 64-wide MN-major box
constexpr int A_BYTES = CTA_M * BK * 2;
constexpr int B_BYTES = CTA_N * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int MAX_GROUPS = gg::MAX_GROUPS;
constexpr int NUM_EPI_WARPS = gg::NUM_EPI_WARPS;
constexpr int FIRST_EPI_WARP = gg::FIRST_EPI_WARP;
constexpr int NUM_THREADS = gg::NUM_THREADS;
constexpr int EPI_COLS = TILE_N / 2;        // columns per epilogue warp
constexpr int EPI_CHUNKS = EPI_COLS / 32;
constexpr int TMEM_COLS = 512;

// Operands of the MMA step of an expert's last rows: as the ring's, 64-wide boxes of 16 rows.
constexpr int SIDE_BOX_BYTES = 64 * UMMA_K * 2;
constexpr int SIDE_A_BYTES = CTA_M / 64 * SIDE_BOX_BYTES;
constexpr int SIDE_BYTES = SIDE_A_BYTES + CTA_N / 64 * SIDE_BOX_BYTES;

struct Shared {
  uint64_t full[STAGES];        // CTA 0's counts: one arrival and the bytes of each CTA
  uint64_t empty[STAGES];
  uint64_t side_full[2];        // CTA 0's counts: one arrival of each CTA
  uint64_t side_empty[2];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];       // CTA 0's counts: every epilogue warp of both CTAs
  uint32_t tmem_base;
  int abort;
  int offs[MAX_GROUPS + 1];
  int tiles[MAX_GROUPS + 1];    // exclusive prefix of the 256 x 256 tiles
  int blocks[MAX_GROUPS + 1];   // input gradient: exclusive prefix of the 128-row blocks
};

constexpr int PATCH_BYTES = gg::PATCH_BYTES;
constexpr int SIDE_OFF = STAGES * STAGE_BYTES;
constexpr int PATCH_OFF = SIDE_OFF + 2 * SIDE_BYTES;
constexpr int AUX_OFF = PATCH_OFF + NUM_EPI_WARPS * PATCH_BYTES;
constexpr int SMEM_BYTES = AUX_OFF + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory");

struct Params {
  int num_groups;
  int m;   // weight gradient only
  int n;
  int k;   // input gradient only
  const int* offs;       // null: `one_group` instead
  int one_group[2];
  void* out;
  const void* aux;
  int accumulate;
  int out_fp32;
  void* psum;
  int side_sums;
  const void* psrc;      // weight gradient: the operands again
  const void* qsrc;
  int* status;
};

struct Tile {
  int group;
  int m_tile;
  int n_tile;
  int row_begin;
  int rows;
};

// `hint`: a group at or before the tile's (a role's tiles come in ascending order, and the next one
// is mostly in the same group or in the one after: a binary search was a fifth of a tile's time in
// the weight gradient of 64 experts).
__device__ __forceinline__ Tile decode(const Shared* sh, int n_tiles, int tile, int& hint) {
  int g = hint;
  while (sh->tiles[g + 1] <= tile) ++g;
  hint = g;
  Tile t;
  const int local = tile - sh->tiles[g];
  t.group = g;
  t.m_tile = local / n_tiles;
  t.n_tile = local - t.m_tile * n_tiles;
  t.row_begin = sh->offs[g];
  t.rows = sh->offs[g + 1] - t.row_begin;
  return t;
}

// ------------------------------------------------------------------------------ activations
// The formulas of gg::gelu_parts on eight pairs at a time, one step of all pairs after the other, as
// an epilogue has two warps per scheduler.  The packed instructions halve the issue slots of the FMAs.
// Measured per tile and CTA (K = 512): 5 thousand cycles without activation, 10 with GELU, 9.2 with
// its reciprocals and exponentials left out: the packed FMAs are most of it.
constexpr int PAIRS = 8;
struct GeluPairs {
  ptx::f32x2 half_erfc[PAIRS];   // 0.5 erfc(|x| / sqrt 2)
  ptx::f32x2 gauss[PAIRS];       // exp(-x^2 / 2)
};
__device__ __forceinline__ void gelu_pairs(const ptx::f32x2 (&x)[PAIRS], GeluPairs& g) {
  using namespace ptx;
  auto both = [](float c) { return pack2(c, c); };
  f32x2 t[PAIRS];
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) {
    float a, b, d0, d1, t0, t1;
    unpack2(x[i], a, b);
    unpack2(fma2(pack2(fabsf(a), fabsf(b)), both(0.3275911f * 0.70710678118654752f), both(1.f)), d0, d1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(d0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(d1));
    t[i] = pack2(t0, t1);
  }
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) {
    float e0, e1, g0, g1;
    unpack2(mul2(x[i], mul2(x[i], both(-0.72134752044448170f))), e0, e1);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(g0) : "f"(e0));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(g1) : "f"(e1));
    g.gauss[i] = pack2(g0, g1);
  }
  f32x2 poly[PAIRS];
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) poly[i] = fma2(both(0.5f * 1.061405429f), t[i], both(0.5f * -1.453152027f));
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) poly[i] = fma2(poly[i], t[i], both(0.5f * 1.421413741f));
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) poly[i] = fma2(poly[i], t[i], both(0.5f * -0.284496736f));
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) poly[i] = fma2(poly[i], t[i], both(0.5f * 0.254829592f));
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) poly[i] = mul2(poly[i], t[i]);
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) g.half_erfc[i] = mul2(poly[i], g.gauss[i]);
}

__device__ __forceinline__ ptx::f32x2 gelu_cdf2(ptx::f32x2 x, ptx::f32x2 half_erfc) {
  float a, b, h0, h1, u0, u1;
  ptx::unpack2(x, a, b);
  ptx::unpack2(half_erfc, h0, h1);
  ptx::unpack2(ptx::fma2(half_erfc, ptx::pack2(-1.f, -1.f), ptx::pack2(1.f, 1.f)), u0, u1);
  return ptx::pack2(a >= 0.f ? u0 : h0, b >= 0.f ? u1 : h1);
}

template <int ACT> __device__ __forceinline__ void act_pairs(ptx::f32x2 (&v)[PAIRS]) {
  if (ACT == kActGelu) {
    GeluPairs g;
    gelu_pairs(v, g);
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) v[i] = ptx::mul2(v[i], gelu_cdf2(v[i], g.half_erfc[i]));
  } else {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
      float a, b;
      ptx::unpack2(v[i], a, b);
      v[i] = ptx::pack2(gg::act_fwd<ACT>(a), gg::act_fwd<ACT>(b));
    }
  }
}

// v *= act'(x)
template <int ACT> __device__ __forceinline__ void act_grad_pairs(const ptx::f32x2 (&x)[PAIRS], ptx::f32x2 (&v)[PAIRS]) {
  if (ACT == kActGelu) {
    GeluPairs g;
    gelu_pairs(x, g);
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
      const ptx::f32x2 d = ptx::fma2(ptx::mul2(x[i], ptx::pack2(0.3989422804014327f, 0.3989422804014327f)), g.gauss[i],
                                     gelu_cdf2(x[i], g.half_erfc[i]));
      v[i] = ptx::mul2(v[i], d);
    }
  } else {
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) {
      float x0, x1, a, b;
      ptx::unpack2(x[i], x0, x1);
      ptx::unpack2(v[i], a, b);
      v[i] = ptx::pack2(gg::act_bwd<ACT>(a, x0), gg::act_bwd<ACT>(b, x1));
    }
  }
}

// ------------------------------------------------------------------------------ epilogue
struct EpiTile {
  uint32_t t_row;           // TMEM address: this warp's lane quarter, first column of its span
  int lane;
  int n_chunks;             // valid 32-column chunks of the span (0..4)
  int warp_valid;           // valid rows of the warp's 32
  uint8_t* patch;
  uint8_t* out;             // first row, first column of the span
  long out_pitch;
  const uint8_t* pre_tile;  // DACT: this warp's 4 x 2 KB of the tile-blocked pre-activation
  uint32_t empty_bar;       // CTA 0's accumulator-free barrier
  const CUtensorMap* map;   // output, boxes of 32 rows x 64 columns; null: not all 32 rows may be written
  int x, y, z;              // first column, row and matrix of the span there
};

// One 32-column chunk, multiplied by the activation's derivative (DACT), into the patch.
template <typename T, int ACT, bool DACT>
__device__ __forceinline__ void finish_chunk(const EpiTile& et, int i, const uint32_t (&r)[32], const Packed32& side) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    ptx::f32x2 v[PAIRS];
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) v[j] = ptx::pack2(__uint_as_float(r[q * 16 + 2 * j]), __uint_as_float(r[q * 16 + 2 * j + 1]));
    if (DACT) {
      ptx::f32x2 x[PAIRS];
#pragma unroll
      for (int j = 0; j < PAIRS; ++j) {
        float a, b;
        Cvt<T>::unpack(side.w[q * 8 + j], a, b);
        x[j] = ptx::pack2(a, b);
      }
      act_grad_pairs<ACT>(x, v);
    }
    uint32_t wo[PAIRS];
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
      float a, b;
      ptx::unpack2(v[j], a, b);
      wo[j] = Cvt<T>::pack(a, b);
    }
    const int c = (i & 1) * 4 + q * 2;
    *reinterpret_cast<uint4*>(gg::patch_piece(et.patch, et.lane, c)) = make_uint4(wo[0], wo[1], wo[2], wo[3]);
    *reinterpret_cast<uint4*>(gg::patch_piece(et.patch, et.lane, c + 1)) = make_uint4(wo[4], wo[5], wo[6], wo[7]);
  }
}

// After an odd chunk (or the last one) the patch holds whole 128-byte lines.  Its swizzle is that of a
// tensor map, so one copy takes all 32 rows (what lies outside the matrix is not written); rows of
// which the last ones belong to the next expert are stored one by one, 8 lanes per row.  Loads from
// the patch and stores were 2.5 of the 5 thousand cycles of a plain tile's epilogue: 22528 rows, 8
// experts, 512 -> 2048, forward and input gradient, with GELU 72 and 72 us, now 67 and 66; with ReLU 59
// and 62, now 55 and 52 (its instances no longer spill either).
__device__ __forceinline__ void send_lines(const EpiTile& et, int i) {
  if (!(i + 1 == et.n_chunks || (i & 1))) return;
  if (et.map != nullptr) {
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (et.lane == 0) {
      ptx::tma_store_3d(et.map, et.patch, et.x + (i & ~1) * 32, et.y, et.z);
      ptx::bulk_commit();
    }
    return;
  }
  const int bytes = ((i & 1) + 1) * 64;
  const int sub = et.lane & 7;
  uint8_t* dst = et.out + (i & ~1) * 64 + sub * 16 + (et.lane >> 3) * et.out_pitch;
  __syncwarp();
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int row = 4 * it + (et.lane >> 3);
    if (row < et.warp_valid && sub * 16 < bytes) {
      *reinterpret_cast<uint4*>(dst + it * 4 * et.out_pitch) =
          *reinterpret_cast<const uint4*>(gg::patch_piece(et.patch, row, sub));
    }
  }
  __syncwarp();
}

// Before the patch is written again: the copies out of it have read it.
__device__ __forceinline__ void patch_free(const EpiTile& et) {
  if (et.lane == 0) ptx::bulk_wait_read<0>();
  __syncwarp();
}

__device__ __forceinline__ void release_accumulator(const EpiTile& et) {
  ptx::tc_fence_before_sync();
  __syncwarp();
  if (et.lane == 0) ptx::mbar_arrive_cluster(et.empty_bar);
}

// One tile for one epilogue warp: the tcgen05.ld of chunk i + 1 (and the load of its saved
// pre-activation) is in flight while chunk i is finished.
template <typename T, int ACT, bool DACT>
__device__ __forceinline__ void epilogue_tile(const EpiTile& et, Packed32& side_a) {
  uint32_t ra[32], rb[32];
  Packed32 side_b;
  bool released = false;
  if (et.n_chunks > 0 && et.warp_valid > 0) {
    ptx::tmem_ld_32x32(et.t_row, ra);
#pragma unroll 1
    for (int i = 0; i < et.n_chunks; i += 2) {
      ptx::tmem_ld_wait();
      const bool second = i + 1 < et.n_chunks;
      if (second) {
        ptx::tmem_ld_32x32(et.t_row + (i + 1) * 32, rb);
        if (DACT) gg::load_pre_chunk(et.pre_tile, i + 1, et.lane, side_b);
      } else {
        release_accumulator(et);
        released = true;
      }
      patch_free(et);
      finish_chunk<T, ACT, DACT>(et, i, ra, side_a);
      send_lines(et, i);
      if (!second) break;
      ptx::tmem_ld_wait();
      if (i + 2 < et.n_chunks) {
        ptx::tmem_ld_32x32(et.t_row + (i + 2) * 32, ra);
        if (DACT) gg::load_pre_chunk(et.pre_tile, i + 2, et.lane, side_a);
      } else {
        release_accumulator(et);
        released = true;
      }
      finish_chunk<T, ACT, DACT>(et, i + 1, rb, side_b);
      send_lines(et, i + 1);
    }
  }
  if (!released) release_accumulator(et);
}

// Weight gradient into an fp32 buffer, or added to the old gradient: the sum is formed in fp32
// from the accumulator, 32-byte accesses per lane and row.
template <typename T>
__device__ __forceinline__ void epilogue_tile_update(const Params& p, const EpiTile& et, long first_elem) {
  uint32_t r[32];
  const bool row_ok = et.lane < et.warp_valid;
  for (int i = 0; i < et.n_chunks && et.warp_valid > 0; ++i) {
    ptx::tmem_ld_32x32(et.t_row + i * 32, r);
    ptx::tmem_ld_wait();
    if (row_ok) {
      const long off = first_elem + static_cast<long>(et.lane) * p.n + i * 32;
      if (p.out_fp32) {
        float* dst = static_cast<float*>(p.out) + off;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w[8];
          if (p.accumulate) gg::ld256(dst + q * 8, w);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float v = __uint_as_float(r[q * 8 + j]);
            w[j] = __float_as_uint(p.accumulate ? __uint_as_float(w[j]) + v : v);
          }
          gg::st256(dst + q * 8, w);
        }
      } else {
        T* dst = static_cast<T*>(p.out) + off;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t w[8];
          gg::ld256(dst + q * 16, w);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float a, b;
            Cvt<T>::unpack(w[j], a, b);
            w[j] = Cvt<T>::pack(a + __uint_as_float(r[q * 16 + 2 * j]), b + __uint_as_float(r[q * 16 + 2 * j + 1]));
          }
          gg::st256(dst + q * 16, w);
        }
      }
    }
    __syncwarp();
  }
  release_accumulator(et);
}

// The bias gradient of a grouped linear is the column sum, per expert, of the matrix its weight gradient
// takes as P.  Either (`side_sums` = 0) on the tiles of the first N column block the epilogue warps, which
// wait for the main loop then, add up this CTA's 128 columns of P with plain 16-byte loads (the rows pass
// through the L2 for the TMA loads at the same time).
template <typename T>
__device__ __forceinline__ void column_sums(const Params& p, uint8_t* patches, const Tile& c, int col0, int warp, int lane) {
  const int ew = warp - FIRST_EPI_WARP;
  const int col = col0 + (lane & 15) * 8;
  const int row_end = c.row_begin + c.rows;
  float cs[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) cs[q] = 0.f;
  auto add = [&](const uint4& v) {
    float a, b;
    Cvt<T>::unpack(v.x, a, b); cs[0] += a; cs[1] += b;
    Cvt<T>::unpack(v.y, a, b); cs[2] += a; cs[3] += b;
    Cvt<T>::unpack(v.z, a, b); cs[4] += a; cs[5] += b;
    Cvt<T>::unpack(v.w, a, b); cs[6] += a; cs[7] += b;
  };
  if (col < p.m) {
    const T* src = static_cast<const T*>(p.psrc) + col;
    int r = c.row_begin + ew * 2 + (lane >> 4);
    constexpr int kUnroll = 16;
    for (; r + 16 * (kUnroll - 1) < row_end; r += 16 * kUnroll) {
      uint4 v[kUnroll];
#pragma unroll
      for (int i = 0; i < kUnroll; ++i) v[i] = __ldg(reinterpret_cast<const uint4*>(src + static_cast<long>(r + 16 * i) * p.m));
#pragma unroll
      for (int i = 0; i < kUnroll; ++i) add(v[i]);
    }
    // (one load after the other, the last 255 rows took 16 times the latency of a load)
    constexpr int kRest = 8;
    for (; r < row_end; r += 16 * kRest) {
      uint4 v[kRest];
#pragma unroll
      for (int i = 0; i < kRest; ++i) {
        v[i] = make_uint4(0u, 0u, 0u, 0u);
        if (r + 16 * i < row_end) v[i] = __ldg(reinterpret_cast<const uint4*>(src + static_cast<long>(r + 16 * i) * p.m));
      }
#pragma unroll
      for (int i = 0; i < kRest; ++i) add(v[i]);
    }
  }
  float* mine = reinterpret_cast<float*>(patches + ew * PATCH_BYTES);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    cs[q] += __shfl_xor_sync(0xffffffffu, cs[q], 16);
    if (lane < 16) mine[lane * 8 + q] = cs[q];
  }
  asm volatile("bar.sync 2, %0;" ::"n"(NUM_EPI_WARPS * 32) : "memory");
  const int tid = static_cast<int>(threadIdx.x) - FIRST_EPI_WARP * 32;
  if (tid < CTA_M && col0 + tid < p.m) {
    float total = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < NUM_EPI_WARPS; ++w8) total += reinterpret_cast<const float*>(patches + w8 * PATCH_BYTES)[tid];
    T* dst = static_cast<T*>(p.psum) + static_cast<long>(c.group) * p.m + col0 + tid;
    if (p.accumulate) total += Cvt<T>::to_f(*dst);
    *dst = Cvt<T>::from_f(total);
  }
  asm volatile("bar.sync 2, %0;" ::"n"(NUM_EPI_WARPS * 32) : "memory");
}

// Or 32 columns at a time by the warps that have little else to do, beside the main loops.  The
// epilogue warps wait for the loads' latency on every tile of the first column block: what the sums add,
// 1024 <-> 4096, 16 experts of 64 rows 9.6 us, here 1 to 3, of 128 rows 8.7, here 0.5; 8 of 2048 rows 10.1, here 3.
// (64 columns at a time and 32 loads in flight took two to three times as long.)  The rule between the two
// is sums_beside() in grouped_gemm.cu.
constexpr int SUM_COLS = 32;
template <typename T>
__device__ __forceinline__ void side_sums(const Params& p, const Shared* sh, int worker, int workers, int lane) {
  const int blocks = (p.m + SUM_COLS - 1) / SUM_COLS;
  auto add = [](float (&cs)[8], const uint4& v) {
    float a, b;
    Cvt<T>::unpack(v.x, a, b); cs[0] += a; cs[1] += b;
    Cvt<T>::unpack(v.y, a, b); cs[2] += a; cs[3] += b;
    Cvt<T>::unpack(v.z, a, b); cs[4] += a; cs[5] += b;
    Cvt<T>::unpack(v.w, a, b); cs[6] += a; cs[7] += b;
  };
  long item = worker;
  for (int g = 0; g < p.num_groups; ++g) {
    const int begin = sh->offs[g], end = sh->offs[g + 1];
    if (end == begin) continue;
    for (; item < blocks; item += workers) {
      const int col = static_cast<int>(item) * SUM_COLS + (lane & 3) * 8;
      float cs[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) cs[q] = 0.f;
      if (col < p.m) {
        const T* src = static_cast<const T*>(p.psrc) + col;
        constexpr int kUnroll = 16;
        for (int r = begin + (lane >> 2); r < end; r += 8 * kUnroll) {
          uint4 v[kUnroll];
#pragma unroll
          for (int i = 0; i < kUnroll; ++i) {
            v[i] = make_uint4(0u, 0u, 0u, 0u);
            if (r + 8 * i < end) v[i] = __ldg(reinterpret_cast<const uint4*>(src + static_cast<long>(r + 8 * i) * p.m));
          }
#pragma unroll
          for (int i = 0; i < kUnroll; ++i) add(cs, v[i]);
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) cs[q] += __shfl_xor_sync(0xffffffffu, cs[q], o);
      }
      if (lane < 4 && col < p.m) {
        T* dst = static_cast<T*>(p.psum) + static_cast<long>(g) * p.m + col;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (p.accumulate) cs[q] += Cvt<T>::to_f(dst[q]);
          dst[q] = Cvt<T>::from_f(cs[q]);
        }
      }
    }
    item -= blocks;
  }
}

// ------------------------------------------------------------------------------ kernel
template <int MODE, typename T, int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + AUX_OFF);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x) >> 1;
  const int num_pairs = static_cast<int>(gridDim.x) >> 1;
  const int n_tiles = (p.n + TILE_N - 1) / TILE_N;
  const int m_tiles_w = (p.m + TILE_M - 1) / TILE_M;
  const volatile int* abort_flag = &sh->abort;

  // ---------------------------------------------------------------- set-up
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&sh->full[s], 2);
      ptx::mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&sh->side_full[b], 2);
      ptx::mbar_init(&sh->side_empty[b], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&sh->tmem_full[a], 1);
      ptx::mbar_init(&sh->tmem_empty[a], 2 * NUM_EPI_WARPS);
    }
    sh->abort = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&tm_a);
    ptx::prefetch_tmap(&tm_b);
    ptx::prefetch_tmap(&tm_c);
  }
  if (warp == 1) ptx::tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
  ptx::chain_begin();   // nothing an earlier kernel writes is read above
  if (warp == 2) {
    // offsets and the prefixes of tiles and blocks; an expert without rows has no tile
    const int* offs = p.offs != nullptr ? p.offs : p.one_group;
    int run = 0, run_b = 0;
    if (lane == 0) {
      sh->tiles[0] = 0;
      sh->blocks[0] = 0;
      sh->offs[0] = offs[0];
    }
    for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
      const int g = g0 + lane;
      int rows = 0, end = 0;
      if (g < p.num_groups) {
        end = offs[g + 1];
        rows = end - offs[g];
      }
      int t = (MODE == kWgrad) ? (rows > 0 ? m_tiles_w * n_tiles : 0) : (rows + TILE_M - 1) / TILE_M * n_tiles;
      int b = (rows + CTA_M - 1) / CTA_M;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int tu = __shfl_up_sync(0xffffffffu, t, o), bu = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
          t += tu;
          b += bu;
        }
      }
      if (g < p.num_groups) {
        sh->offs[g + 1] = end;
        sh->tiles[g + 1] = run + t;
        sh->blocks[g + 1] = run_b + b;
      }
      run += __shfl_sync(0xffffffffu, t, 31);
      run_b += __shfl_sync(0xffffffffu, b, 31);
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync();
  ptx::tc_fence_after_sync();

  const uint32_t tmem_base = sh->tmem_base;
  const int total = sh->tiles[p.num_groups];
  int group = 0;   // of the role's latest tile

  if (warp == 0) {
    // ============================================================== TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < total && ok; tile += num_pairs) {
        const Tile c = decode(sh, n_tiles, tile, group);
        const int num_kb = (MODE == kWgrad) ? (c.rows / UMMA_K * UMMA_K + BK - 1) / BK : p.k / BK;
        const int n0 = c.n_tile * TILE_N + rank * CTA_N;
        const int m0 = c.m_tile * TILE_M + rank * CTA_M;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          const uint32_t bar = ptx::mapa(&sh->full[stage], 0);
          ptx::mbar_arrive_expect_tx_cluster(bar, STAGE_BYTES);
          if (MODE == kRowsNN) {
            ptx::tma_load_2d_pair(sa, &tm_a, bar, kb * BK, c.row_begin + m0);
#pragma unroll
            for (int ch = 0; ch < CTA_N / 64; ++ch) {
              ptx::tma_load_2d_pair(sb + ch * BOX_BYTES, &tm_b, bar, n0 + ch * 64, c.group * p.k + kb * BK);
            }
          } else {
            const int row0 = c.row_begin + kb * BK;
#pragma unroll
            for (int ch = 0; ch < CTA_M / 64; ++ch) ptx::tma_load_2d_pair(sa + ch * BOX_BYTES, &tm_a, bar, m0 + ch * 64, row0);
#pragma unroll
            for (int ch = 0; ch < CTA_N / 64; ++ch) ptx::tma_load_2d_pair(sb + ch * BOX_BYTES, &tm_b, bar, n0 + ch * 64, row0);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ============================================================== MMA issuer (CTA 0)
    if (rank == 0 && lane == 0) {
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t idesc = ptx::make_idesc(kBf16, MODE == kWgrad, true, TILE_M, TILE_N);
      int stage = 0;
      uint32_t phase = 0;
      int iter = 0, side = 0;
      bool ok = true;
      for (int tile = pair; tile < total && ok; tile += num_pairs, ++iter) {
        const Tile c = decode(sh, n_tiles, tile, group);
        const int whole = c.rows / UMMA_K * UMMA_K;   // rows in full MMA steps (weight gradient)
        const int num_kb = (MODE == kWgrad) ? (whole + BK - 1) / BK : p.k / BK;
        const int acc = iter & 1;
        if (!ptx::mbar_wait(&sh->tmem_empty[acc], ((iter >> 1) & 1) ^ 1, abort_flag)) {
          sh->abort = 1;
          if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * TILE_N;
        const bool ragged = MODE == kWgrad && whole != c.rows;
        if (ragged) {   // first: its operands have been there for long, and the ring goes on filling
          if (!ptx::mbar_wait<true>(&sh->side_full[side & 1], (side >> 1) & 1, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sa = ptx::smem_u32(smem + SIDE_OFF + (side & 1) * SIDE_BYTES);
          const uint64_t a_desc = ptx::make_smem_desc_sw128(sa, SIDE_BOX_BYTES, 1024);
          const uint64_t b_desc = ptx::make_smem_desc_sw128(sa + SIDE_A_BYTES, SIDE_BOX_BYTES, 1024);
          ptx::umma_f16_pair(d_tmem, a_desc, b_desc, idesc, 0u);
          ptx::umma_commit_pair(&sh->side_empty[side & 1]);
          ++side;
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&sh->full[stage], phase, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sa = ptx::smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          const int steps = (MODE == kWgrad) ? min(BK / UMMA_K, (whole - kb * BK) / UMMA_K) : BK / UMMA_K;
#pragma unroll
          for (int k16 = 0; k16 < BK / UMMA_K; ++k16) {
            if (MODE == kWgrad && k16 >= steps) break;
            // K-major operands: 32 bytes per K step inside the 128-byte swizzle row; MN-major
            // operands: 16 K rows per step, 64-wide boxes 8 KB apart
            const uint64_t a_desc = (MODE == kWgrad)
                ? ptx::make_smem_desc_sw128(sa + k16 * (UMMA_K * 128), BOX_BYTES, 1024)
                : ptx::make_smem_desc_sw128(sa + k16 * (UMMA_K * 2), 16, 1024);
            const uint64_t b_desc = ptx::make_smem_desc_sw128(sb + k16 * (UMMA_K * 128), BOX_BYTES, 1024);
            ptx::umma_f16_pair(d_tmem, a_desc, b_desc, idesc, (kb | k16) != 0 || ragged ? 1u : 0u);
          }
          ptx::umma_commit_pair(&sh->empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        ptx::umma_commit_pair(&sh->tmem_full[acc]);
      }
    }
  } else if (warp == 2) {
    // ============================================================== ragged ends
    if constexpr (MODE == kWgrad) {
      static_assert((CTA_M + CTA_N) / 64 * 8 == 32, "16 bytes of a row per lane");
      const int box = lane >> 3, chunk = lane & 7;
      const bool of_a = box < CTA_M / 64;
      const long pitch = of_a ? p.m : p.n;
      int side = 0;
      for (int tile = pair; tile < total; tile += num_pairs) {
        const Tile c = decode(sh, n_tiles, tile, group);
        const int rest = c.rows % UMMA_K;
        if (rest == 0) continue;
        const int col = (of_a ? c.m_tile * TILE_M + rank * CTA_M + box * 64
                              : c.n_tile * TILE_N + rank * CTA_N + (box - CTA_M / 64) * 64) + chunk * 8;
        const T* src = static_cast<const T*>(of_a ? p.psrc : p.qsrc) + (static_cast<long>(c.row_begin) + c.rows - rest) * pitch + col;
        uint4 v[UMMA_K - 1];
#pragma unroll
        for (int r = 0; r < UMMA_K - 1; ++r) {
          v[r] = make_uint4(0u, 0u, 0u, 0u);
          if (r < rest && col < pitch) v[r] = __ldg(reinterpret_cast<const uint4*>(src + r * pitch));
        }
        if (!ptx::mbar_wait(&sh->side_empty[side & 1], ((side >> 1) & 1) ^ 1, abort_flag)) {
          if (lane == 0) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_PRODUCER);
          }
          break;
        }
        // 128-byte swizzle: the 16-byte chunks of row r change places by r % 8
        uint8_t* at = smem + SIDE_OFF + (side & 1) * SIDE_BYTES + box * SIDE_BOX_BYTES;
#pragma unroll
        for (int r = 0; r < UMMA_K; ++r) {
          *reinterpret_cast<uint4*>(at + r * 128 + ((chunk ^ (r & 7)) << 4)) = r < UMMA_K - 1 ? v[r < UMMA_K - 1 ? r : 0] : make_uint4(0u, 0u, 0u, 0u);
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_release_cluster(ptx::mapa(&sh->side_full[side & 1], 0));
        ++side;
      }
    }
  } else if (warp == 3) {
    // ============================================================== experts without rows
    if constexpr (MODE == kWgrad) {
      if (!p.accumulate) {
        const long bytes = static_cast<long>(p.m) * p.n * (p.out_fp32 ? 4 : 2);   // a multiple of 512
        const uint32_t zero[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        for (int g = 0; g < p.num_groups; ++g) {
          if (sh->offs[g + 1] != sh->offs[g]) continue;
          uint8_t* dst = static_cast<uint8_t*>(p.out) + g * bytes;
          for (long i = (static_cast<long>(blockIdx.x) * 32 + lane) * 32; i < bytes; i += static_cast<long>(gridDim.x) * 1024) {
            gg::st256(dst + i, zero);
          }
          if (p.psum != nullptr && g % static_cast<int>(gridDim.x) == static_cast<int>(blockIdx.x)) {
            T* ps = static_cast<T*>(p.psum) + static_cast<long>(g) * p.m;
            for (int i = lane; i < p.m; i += 32) ps[i] = Cvt<T>::from_f(0.f);
          }
        }
      }
      if (p.psum != nullptr && p.side_sums) side_sums<T>(p, sh, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x), lane);
    }
  } else {
    // ============================================================== epilogue (warps 4..11)
    const int part = warp & 3;                       // TMEM lane quarter this warp may read
    const int half = (warp - FIRST_EPI_WARP) >> 2;   // which half of the accumulator columns
    const int ew = warp - FIRST_EPI_WARP;
    uint8_t* patches = smem + PATCH_OFF;
    int iter = 0;
    bool dead = false;   // a wait ran out: walk the remaining tiles' barriers, touch nothing else
    for (int tile = pair; tile < total; tile += num_pairs, ++iter) {
      const Tile c = decode(sh, n_tiles, tile, group);
      const int acc = iter & 1;
      const int col_first = c.n_tile * TILE_N + half * EPI_COLS;
      const int m0 = c.m_tile * TILE_M + rank * CTA_M + part * 32;
      EpiTile et;
      et.lane = lane;
      et.n_chunks = max(0, min(EPI_CHUNKS, (p.n - col_first) / 32));
      et.warp_valid = max(0, min(32, ((MODE == kWgrad) ? p.m : c.rows) - m0));
      et.patch = patches + ew * PATCH_BYTES;
      et.out_pitch = static_cast<long>(p.n) * 2;
      et.pre_tile = nullptr;
      et.empty_bar = ptx::mapa(&sh->tmem_empty[acc], 0);
      et.t_row = tmem_base + (static_cast<uint32_t>(part * 32) << 16) + acc * TILE_N + half * EPI_COLS;
      const long first_elem = ((MODE == kWgrad) ? static_cast<long>(c.group) * p.m + m0 : static_cast<long>(c.row_begin) + m0) * p.n + col_first;
      et.out = static_cast<uint8_t*>(p.out) + first_elem * 2;
      et.map = MODE == kWgrad || et.warp_valid == 32 ? &tm_c : nullptr;
      et.x = col_first;
      et.y = MODE == kWgrad ? m0 : c.row_begin + m0;
      et.z = MODE == kWgrad ? c.group : 0;
      Packed32 side;
      if constexpr (MODE == kWgrad) {
        if (p.psum != nullptr && !p.side_sums && c.n_tile == 0) {
          patch_free(et);
          column_sums<T>(p, patches, c, c.m_tile * TILE_M + rank * CTA_M, warp, lane);
        }
      } else {
        // the tile-blocked layout counts 128 x 256 blocks, groups in order
        const long blk = (static_cast<long>(sh->blocks[c.group]) + c.m_tile * 2 + rank) * n_tiles + c.n_tile;
        et.pre_tile = static_cast<const uint8_t*>(p.aux) + blk * gg::PRE_TILE_BYTES + ew * (gg::CHUNKS_PER_WARP * gg::PRE_CHUNK_BYTES);
        if (et.n_chunks > 0 && et.warp_valid > 0) {
          // it does not depend on the accumulator: fetch the first chunk before the wait, and
          // pull the next tile's chunks of this warp (8 KB, two lines per lane) into L2
          gg::load_pre_chunk(et.pre_tile, 0, lane, side);
          if (tile + num_pairs < total) {
            int ahead = group;
            const Tile cn = decode(sh, n_tiles, tile + num_pairs, ahead);
            if (cn.m_tile * TILE_M + rank * CTA_M < cn.rows) {
              const long nb = (static_cast<long>(sh->blocks[cn.group]) + cn.m_tile * 2 + rank) * n_tiles + cn.n_tile;
              const uint8_t* nx = static_cast<const uint8_t*>(p.aux) + nb * gg::PRE_TILE_BYTES +
                                  ew * (gg::CHUNKS_PER_WARP * gg::PRE_CHUNK_BYTES) + lane * 256;
              asm volatile("prefetch.global.L2 [%0];" ::"l"(nx));
              asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + 128));
            }
          }
        }
      }
      if (dead) continue;
      if (!ptx::mbar_wait(&sh->tmem_full[acc], (iter >> 1) & 1, abort_flag)) {
        if (lane == 0) {
          sh->abort = 1;
          if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_EPILOGUE);
        }
        dead = true;
        continue;
      }
      ptx::tc_fence_after_sync();
      if (MODE == kWgrad && (p.out_fp32 || p.accumulate)) {
        epilogue_tile_update<T>(p, et, first_elem);
      } else {
        epilogue_tile<T, ACT, MODE == kRowsNN>(et, side);
      }
      __syncwarp();
    }
  }

  // ---------------------------------------------------------------- tear-down
  if (lane == 0) ptx::bulk_wait<0>();
  __syncwarp();
  if (*abort_flag != 0) {
    // give copies that were already issued time to land before the shared memory goes away
    const unsigned long long t0 = ptx::globaltimer();
    while (ptx::globaltimer() - t0 < 200000ull) __nanosleep(1000);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync();   // the other CTA may still signal this CTA's barriers until here
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------ launch
template <int MODE, typename T, int ACT>
cudaError_t launch_one(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p, int grid, cudaStream_t stream) {
  static std::mutex mu;   // the shared-memory attribute is per device
  static uint64_t configured = 0;
  auto kernel = pair_gemm_kernel<MODE, T, ACT>;
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!(configured >> (dev & 63) & 1)) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
      if (e != cudaSuccess) return e;
      configured |= 1ull << (dev & 63);
    }
  }
  return launch_chained(kernel, dim3(grid), dim3(NUM_THREADS), SMEM_BYTES, stream, ta, tb, tc, p);
}

// One translation unit per element type instantiates this.
template <typename T>
cudaError_t launch_for_type(int mode, int act, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p,
                            int grid, cudaStream_t stream) {
  if (mode == kWgrad) return launch_one<kWgrad, T, kActNone>(ta, tb, tc, p, grid, stream);
  switch (act) {
    case kActRelu: return launch_one<kRowsNN, T, kActRelu>(ta, tb, tc, p, grid, stream);
    case kActGelu: return launch_one<kRowsNN, T, kActGelu>(ta, tb, tc, p, grid, stream);
    case kActGeluTanh: return launch_one<kRowsNN, T, kActGeluTanh>(ta, tb, tc, p, grid, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_bf16(int mode, int act, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p, int grid,
                        cudaStream_t stream);
cudaError_t launch_f16(int mode, int act, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p, int grid,
                       cudaStream_t stream);

}  // namespace pg
}  // namespace fmoe
