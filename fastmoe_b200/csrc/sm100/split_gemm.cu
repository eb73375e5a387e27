// fp32 grouped GEMM on the tensor cores.
//
// An fp32 value is the sum of three bf16 values, h + m + l (8 + 8 + 8 bits, each the rounded rest of
// the one before), so that a product of two is the sum of nine bf16 products, each exact in fp32.  Six are
// formed: h h, and the five of the next two orders (h m, m h, and m m, h l, l h); what is left out (m l,
// l m, l l) is below 2^-26 of the product.  tf32, the tensor cores' own fp32 format, would drop 13 bits of
// the inputs instead.  m and l are held as m 2^7 and l 2^14, which keeps them in bf16's range where
// the value is in fp32's, but for an error of at most 2^-148; unscaled, the rests of a value below 2^-110 fall
// under the smallest bf16 subnormal, 2^-133 (at 2^-120 6e-5 of the value was lost).  Larger scales would let the
// small products overflow before the result does.  The three orders have an accumulator each.
//
// The tensor cores add with truncation, which over a long sum costs more than the roundings of fp32
// FMAs.  So h h is accumulated in TMEM over one K block of 64 only (four additions); the epilogue
// warps take every block's sum into registers and add them in fp32, rounded to nearest.  The small
// products are accumulated over the whole sum: they are 2^-8 of the result and less.
// Keeping them apart also keeps infinities: inf - inf of h l and h m would be NaN where the
// product is inf, so a total that is not finite is replaced by the sum of h h.
//
// Error against 64 bits (2-norm, 8 experts, 4096 rows, 512 -> 2048): forward 9.0e-8, input gradient
// 1.1e-7, weight gradient 9.0e-8, where FMAs in ascending order have 4.1e-7, 8.1e-7 and 4.1e-7.
//
// What bounds it: the tensor cores, at six times the bf16 work, and the shared memory their operands
// come from.  4 experts, 16384 rows, 1024 -> 2048: 307 to 327 us = 1260 to 1340 TFLOP/s of bf16
// products, 210 to 224 of fp32, with the splitting 355 to 417, where the FMA kernel (sgemm.cu) takes
// 1290 to 1400.  A plane of A serves all its products in a row out of the operand collector: 4 to 5 %.
// A pair of CTAs (cta_group::2) works on a 256 x 128 tile, half the width of the 16-bit kernel's: an
// epilogue warp holds 32 x 64 sums in registers, 64 per thread, and fp32 layers are small (512 outputs
// of 8 experts with 512 rows are 64 such tiles for 74 pairs).  The tiles of the last round are cut along
// K (tile_walk.cuh): 8 experts with 384 to 640 rows, 2048 -> 512, 121 against 141 us, splitting included.
//
// Roles of a CTA (384 threads), persistent over the tiles of its pair:
//   warp 0      TMA producer, one lane: three planes of this CTA's halves of A and B per K block, 72 KB
//               a stage, 3 stages;
//   warp 1      CTA 0: one lane issues the MMAs; in both CTAs the warp owns the TMEM allocation;
//   warps 2, 3  weight gradient: column sums of P (the bias gradient) and zeros of experts without
//               rows; row modes: zeros past the last expert;
//   warps 4-11  epilogue.
// TMEM: two accumulators of 128 columns for h h in turn, one each for the products of the next two orders.
// (One for both of these, unscaled, leaves three for h h: what an epilogue with an activation holds up is a
// K block less then.  8 experts, 4096 rows, 512 -> 2048: GELU 103 -> 106 us, its derivative 106 -> 116, plain
// products the same to 3 %; the scales are worth it, see above.)
#include "split_gemm.cuh"

#include <float.h>

#include <mutex>

#include "grouped_gemm.cuh"
#include "grouped_gemm_kernel.cuh"
#include "launch.cuh"
#include "ptx.cuh"
#include "tensor_map.cuh"
#include "tile_walk.cuh"

namespace fmoe {
namespace {

using bf16 = __nv_bfloat16;

constexpr int CTA_M = 128;
constexpr int TILE_M = 2 * CTA_M;
constexpr int TILE_N = 128;
constexpr int CTA_N = TILE_N / 2;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int STAGES = 3;
constexpr int BOX_BYTES = 64 * BK * 2;
constexpr int A_BYTES = CTA_M * BK * 2;          // one plane
constexpr int B_BYTES = CTA_N * BK * 2;
constexpr int B_OFF = 3 * A_BYTES;
constexpr int STAGE_BYTES = 3 * (A_BYTES + B_BYTES);
constexpr int MAX_GROUPS = gg::MAX_GROUPS;
constexpr int NUM_EPI_WARPS = 8;
constexpr int FIRST_EPI_WARP = 4;
constexpr int NUM_THREADS = (FIRST_EPI_WARP + NUM_EPI_WARPS) * 32;
constexpr int EPI_COLS = TILE_N / 2;             // columns per epilogue warp
constexpr int MAIN_BUFS = 2;
constexpr int M_COL = MAIN_BUFS * TILE_N;        // TMEM columns of the products with one m, and of the order after
constexpr int L_COL = M_COL + TILE_N;
constexpr int TMEM_COLS = 512;
constexpr float M_SCALE = 128.f, L_SCALE = M_SCALE * M_SCALE;   // (m m is of l's order)

struct Shared {
  uint64_t full[STAGES];          // CTA 0's counts: one arrival and the bytes of each CTA
  uint64_t empty[STAGES];
  uint64_t main_full[MAIN_BUFS];
  uint64_t main_empty[MAIN_BUFS];  // CTA 0's counts: every epilogue warp of both CTAs
  uint64_t small_full;
  uint64_t small_empty;
  uint32_t tmem_base;
  int abort;
  int offs[MAX_GROUPS + 1];
  int tiles[MAX_GROUPS + 1];      // exclusive prefixes of the tiles and of their K blocks
  int units[MAX_GROUPS + 1];
};
constexpr int AUX_OFF = STAGES * STAGE_BYTES;
constexpr int SMEM_BYTES = AUX_OFF + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory");

struct Params {
  int num_groups;
  int m, n, k;
  long rows_cap;
  long plane_rows;       // rows per plane of the token matrices
  const int* offs;
  const float* bias;
  float* out;
  bf16* planes;
  float* pre;
  const bf16* psrc;
  float* psum;
  float* work;           // sums of tiles that several pairs share, and their flags (zero before the
  int* flags;            // launch); null: no tile is shared
  float* sums;           // [slots][m] pieces of the column sums, and how many of each expert and
  int* sum_counts;       // 64 columns are there (zero before the launch)
  int* status;
};

// A shared sum: one piece of 32 x 64 per epilogue warp.
constexpr int WORK_FLOATS = 32 * EPI_COLS;
constexpr int COST_KB = 3;   // of 0.8 us: handing a sum over and collecting one takes about 2 us
constexpr unsigned long long COLLECT_LIMIT_NS = 30000000000ull;   // other streams may hold the SMs meanwhile

// Pieces of the column sums: expert e's begin at slot sum_slot(offs[e], e).
constexpr int SUM_ROWS = 256;
__host__ __device__ inline long sum_slot(long off, long e) { return off / SUM_ROWS + 2 * e; }

struct Tile {
  int group, m_tile, n_tile;
  int row_begin, rows;
  long padded;           // first padded row of the group
};

__device__ __forceinline__ Tile decode(const Shared* sh, int n_tiles, const WalkPart& w) {
  Tile t;
  t.group = w.group;
  t.m_tile = w.tile / n_tiles;
  t.n_tile = w.tile - t.m_tile * n_tiles;
  t.row_begin = sh->offs[w.group];
  t.rows = sh->offs[w.group + 1] - t.row_begin;
  t.padded = split_row(t.row_begin, w.group);
  return t;
}

// ------------------------------------------------------------------------------ values
// h + m / M_SCALE + l / L_SCALE == x for finite x, l exact in bf16 for x of at least 2^-124 and rounded to a
// multiple of 2^-133 below; the planes of a value that is not finite are (x, 0, 0).
__device__ __forceinline__ void split1(float x, float& h, float& m, float& l) {
  // 0x7f7f8000 and above would round to infinity: the largest bf16 value is taken instead
  const float mag = fminf(fabsf(x), __uint_as_float(0x7f7f0000u));
  h = __bfloat162float(__float2bfloat16_rn(copysignf(mag, x)));
  const float r = (x - h) * M_SCALE;
  m = __bfloat162float(__float2bfloat16_rn(r));
  l = (r - m) * (L_SCALE / M_SCALE);
  if (!(fabsf(x) <= FLT_MAX)) {
    h = x;
    m = 0.f;
    l = 0.f;
  }
}

// The value again; the sum of the two smaller parts is rounded once.
__device__ __forceinline__ float join3(float h, float m, float l) { return h + fmaf(l, 1.f / L_SCALE, m * (1.f / M_SCALE)); }

__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  float h0, m0, l0, h1, m1, l1;
  split1(a, h0, m0, l0);
  split1(b, h1, m1, l1);
  h = gg::Cvt<bf16>::pack(h0, h1);
  m = gg::Cvt<bf16>::pack(m0, m1);
  l = gg::Cvt<bf16>::pack(l0, l1);
}

// Eight values to 16 bytes of each plane.
__device__ __forceinline__ void store_split8(bf16* dst, long plane, const float (&v)[8]) {
  uint4 w[3];
#pragma unroll
  for (int j = 0; j < 4; ++j) split2(v[2 * j], v[2 * j + 1], (&w[0].x)[j], (&w[1].x)[j], (&w[2].x)[j]);
  *reinterpret_cast<uint4*>(dst) = w[0];
  *reinterpret_cast<uint4*>(dst + plane) = w[1];
  *reinterpret_cast<uint4*>(dst + 2 * plane) = w[2];
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// The activations in full fp32, as torch.nn.functional computes them.
template <int ACT> __device__ __forceinline__ float act32(float x) {
  if (ACT == kActRelu) return gg::relu(x);
  if (ACT == kActGelu) return x * 0.5f * (1.f + erff(x * 0.70710678118654752f));
  if (ACT == kActGeluTanh) {
    const float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return 0.5f * x * (1.f + tanhf(inner));
  }
  return x;
}
template <int ACT> __device__ __forceinline__ float act32_bwd(float g, float x) {
  if (ACT == kActRelu) return x <= 0.f ? 0.f : g;
  if (ACT == kActGelu) {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    const float pdf = expf(-0.5f * x * x) * 0.3989422804014327f;
    return g * (cdf + x * pdf);
  }
  if (ACT == kActGeluTanh) {
    const float x2 = x * x;
    const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x2 * x));
    const float left = 0.5f * x, right = 1.f + t;
    const float d_inner = 0.7978845608028654f * (1.f + 3.f * 0.044715f * x2);
    return g * (0.5f * right + left * (1.f - t * t) * d_inner);
  }
  return g;
}

// ------------------------------------------------------------------------------ kernel
template <int MODE, int KIND, int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
split_gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                  const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + AUX_OFF);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x) >> 1;
  const int num_pairs = static_cast<int>(gridDim.x) >> 1;
  const int n_tiles = (p.n + TILE_N - 1) / TILE_N;
  const int m_tiles_w = (p.m + TILE_M - 1) / TILE_M;   // weight gradient
  const volatile int* abort_flag = &sh->abort;

  // ---------------------------------------------------------------- set-up
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&sh->full[s], 2);
      ptx::mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < MAIN_BUFS; ++b) {
      ptx::mbar_init(&sh->main_full[b], 1);
      ptx::mbar_init(&sh->main_empty[b], 2 * NUM_EPI_WARPS);
    }
    ptx::mbar_init(&sh->small_full, 1);
    ptx::mbar_init(&sh->small_empty, 2 * NUM_EPI_WARPS);
    sh->abort = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&tm_a);
    ptx::prefetch_tmap(&tm_b);
  }
  if (warp == 1) ptx::tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
  ptx::chain_begin();   // nothing an earlier kernel writes is read above
  if (warp == 2) {
    // offsets and the prefixes; an expert without rows has no tile
    int run = 0, run_u = 0;
    if (lane == 0) {
      sh->tiles[0] = 0;
      sh->units[0] = 0;
      sh->offs[0] = p.offs[0];
    }
    for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
      const int g = g0 + lane;
      int rows = 0, end = 0;
      if (g < p.num_groups) {
        end = p.offs[g + 1];
        rows = end - p.offs[g];
      }
      int t = (MODE == kWgrad) ? (rows > 0 ? m_tiles_w * n_tiles : 0) : (rows + TILE_M - 1) / TILE_M * n_tiles;
      int u = t * (((MODE == kWgrad ? rows : p.k) + BK - 1) / BK);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int tu = __shfl_up_sync(0xffffffffu, t, o), uu = __shfl_up_sync(0xffffffffu, u, o);
        if (lane >= o) {
          t += tu;
          u += uu;
        }
      }
      if (g < p.num_groups) {
        sh->offs[g + 1] = end;
        sh->tiles[g + 1] = run + t;
        sh->units[g + 1] = run_u + u;
      }
      run += __shfl_sync(0xffffffffu, t, 31);
      run_u += __shfl_sync(0xffffffffu, u, 31);
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync();
  ptx::tc_fence_after_sync();

  const uint32_t tmem_base = sh->tmem_base;
  TileWalk walk(sh->tiles, sh->units, p.num_groups, pair, num_pairs, p.work != nullptr ? COST_KB : 0);
  WalkPart part_of;

  if (warp == 0) {
    // ============================================================== TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      while (ok && walk.next(part_of)) {
        const Tile c = decode(sh, n_tiles, part_of);
        const int n0 = c.n_tile * TILE_N + rank * CTA_N;
        const int m0 = c.m_tile * TILE_M + rank * CTA_M;
        for (int kb = part_of.kb0; kb < part_of.kb1; ++kb) {
          if (!ptx::mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + B_OFF;
          const uint32_t bar = ptx::mapa(&sh->full[stage], 0);
          ptx::mbar_arrive_expect_tx_cluster(bar, STAGE_BYTES);
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) {
            const int row = static_cast<int>(pl * p.plane_rows + c.padded);
            uint8_t* da = sa + pl * A_BYTES;
            uint8_t* db = sb + pl * B_BYTES;
            if (MODE == kWgrad) {
              ptx::tma_load_2d_pair(da, &tm_a, bar, m0, row + kb * BK);
              ptx::tma_load_2d_pair(da + BOX_BYTES, &tm_a, bar, m0 + 64, row + kb * BK);
              ptx::tma_load_2d_pair(db, &tm_b, bar, n0, row + kb * BK);
            } else {
              ptx::tma_load_2d_pair(da, &tm_a, bar, kb * BK, row + m0);
              if (MODE == kRowsNT) {
                ptx::tma_load_2d_pair(db, &tm_b, bar, kb * BK, (pl * p.num_groups + c.group) * p.n + n0);
              } else {
                ptx::tma_load_3d_pair(db, &tm_b, bar, n0, kb * BK, pl * p.num_groups + c.group);
              }
            }
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ============================================================== MMA issuer (CTA 0)
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc = ptx::make_idesc(true, MODE == kWgrad, MODE != kRowsNT, TILE_M, TILE_N);
      int stage = 0, buf = 0;
      uint32_t phase = 0, buf_phase = 0, small_phase = 0;
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (ptx::mbar_wait(bar, parity, abort_flag)) return true;
        sh->abort = 1;
        if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
        return false;
      };
      while (ok && walk.next(part_of)) {
        const Tile c = decode(sh, n_tiles, part_of);
        const int len = MODE == kWgrad ? c.rows : p.k;
        const uint32_t d_m = tmem_base + M_COL, d_l = tmem_base + L_COL;
        for (int kb = part_of.kb0; kb < part_of.kb1; ++kb) {
          const uint32_t d_main = tmem_base + buf * TILE_N;
          if (!(ok = wait(&sh->main_empty[buf], buf_phase ^ 1) && wait(&sh->full[stage], phase))) break;
          ptx::tc_fence_after_sync();
          const uint32_t sa = ptx::smem_u32(smem + stage * STAGE_BYTES);
          const int steps = min(BK / UMMA_K, (len - kb * BK + UMMA_K - 1) / UMMA_K);
          // K-major operands: 32 bytes per K step inside the 128-byte swizzle row; MN-major
          // operands: 16 K rows per step, 64-wide boxes.  A descriptor's address is its lowest field:
          // planes and K steps are constants added to it.  (An MMA takes 64 cycles; with descriptors
          // formed one by one the issuing thread took longer than that.)
          const uint64_t a0 = MODE == kWgrad ? ptx::make_smem_desc_sw128(sa, BOX_BYTES, 1024) : ptx::make_smem_desc_sw128(sa, 16, 1024);
          const uint64_t b0 = MODE == kRowsNT ? ptx::make_smem_desc_sw128(sa + B_OFF, 16, 1024)
                                              : ptx::make_smem_desc_sw128(sa + B_OFF, BOX_BYTES, 1024);
          constexpr int kStepA = (MODE == kWgrad ? UMMA_K * 128 : UMMA_K * 2) >> 4;
          constexpr int kStepB = (MODE == kRowsNT ? UMMA_K * 2 : UMMA_K * 128) >> 4;
          auto desc_a = [&](int pl, int k16) { return a0 + (pl * (A_BYTES >> 4) + k16 * kStepA); };
          auto desc_b = [&](int pl, int k16) { return b0 + (pl * (B_BYTES >> 4) + k16 * kStepB); };
          const bool first = kb == part_of.kb0;
          if (first) {
            if (!(ok = wait(&sh->small_empty, small_phase ^ 1))) break;
            ptx::tc_fence_after_sync();
          }
          // a plane of A serves all its products in a row
#pragma unroll
          for (int k16 = 0; k16 < BK / UMMA_K; ++k16) {
            if (k16 < steps) {
              ptx::umma_f16_pair_collect<ptx::kCollectFill>(d_main, desc_a(0, k16), desc_b(0, k16), idesc, k16 != 0 ? 1u : 0u);
              const uint32_t on = first && k16 == 0 ? 0u : 1u;
              ptx::umma_f16_pair_collect<ptx::kCollectUse>(d_l, desc_a(0, k16), desc_b(2, k16), idesc, on);
              ptx::umma_f16_pair_collect<ptx::kCollectLast>(d_m, desc_a(0, k16), desc_b(1, k16), idesc, on);
              ptx::umma_f16_pair_collect<ptx::kCollectFill>(d_l, desc_a(1, k16), desc_b(1, k16), idesc, 1u);
              ptx::umma_f16_pair_collect<ptx::kCollectLast>(d_m, desc_a(1, k16), desc_b(0, k16), idesc, 1u);
              ptx::umma_f16_pair(d_l, desc_a(2, k16), desc_b(0, k16), idesc, 1u);
            }
          }
          ptx::umma_commit_pair(&sh->main_full[buf]);
          if (++buf == MAIN_BUFS) { buf = 0; buf_phase ^= 1; }
          ptx::umma_commit_pair(&sh->empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        ptx::umma_commit_pair(&sh->small_full);
        small_phase ^= 1;
      }
    }
  } else if (warp < FIRST_EPI_WARP) {
    const int side = warp - 2;
    if constexpr (MODE == kWgrad) {
      // ============================================================ column sums, empty experts
      if (p.psum != nullptr) {
        // 256 rows x 64 columns of P at a time (8 lanes x 8 columns, 4 x 4 rows per step), dealt out
        // to these two warps of all CTAs; the warp that finishes an expert's columns last adds the
        // pieces up in their order
        const int col_blocks = (p.m + 63) / 64;
        const int last = sh->offs[p.num_groups];
        const long slots = sum_slot(last > 0 ? last - 1 : 0, p.num_groups - 1) + 1;
        const long plane = p.plane_rows * p.m;
        for (long item = static_cast<long>(blockIdx.x) * 2 + side; item < slots * col_blocks; item += static_cast<long>(gridDim.x) * 2) {
          const long slot = item / col_blocks;
          const int cb = static_cast<int>(item - slot * col_blocks);
          int lo = 0, hi = p.num_groups;   // the last expert whose slots begin at or before this one
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (sum_slot(sh->offs[mid], mid) <= slot) lo = mid; else hi = mid;
          }
          const int rows = sh->offs[lo + 1] - sh->offs[lo];
          const long first_slot = sum_slot(sh->offs[lo], lo);
          const int r0 = static_cast<int>(slot - first_slot) * SUM_ROWS;
          if (r0 >= rows) continue;
          const int r1 = min(rows, r0 + SUM_ROWS);
          const int col = cb * 64 + (lane & 7) * 8;
          float cs[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          if (col < p.m) {
            const bf16* src = p.psrc + split_row(sh->offs[lo], lo) * p.m + col;
            constexpr int kUnroll = 4;
            for (int r = r0 + (lane >> 3); r < r1; r += 4 * kUnroll) {
              uint4 v[kUnroll][3];
#pragma unroll
              for (int u = 0; u < kUnroll; ++u) {
#pragma unroll
                for (int pl = 0; pl < 3; ++pl) {
                  v[u][pl] = make_uint4(0u, 0u, 0u, 0u);
                  if (r + 4 * u < r1) v[u][pl] = __ldg(reinterpret_cast<const uint4*>(src + pl * plane + static_cast<long>(r + 4 * u) * p.m));
                }
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {   // the rows of one step among themselves, then to the sum
                float sa = 0.f, sb = 0.f;
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                  float a[3], b[3];
#pragma unroll
                  for (int pl = 0; pl < 3; ++pl) gg::Cvt<bf16>::unpack((&v[u][pl].x)[j], a[pl], b[pl]);
                  sa += join3(a[0], a[1], a[2]);
                  sb += join3(b[0], b[1], b[2]);
                }
                cs[2 * j] += sa;
                cs[2 * j + 1] += sb;
              }
            }
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            cs[q] += __shfl_xor_sync(0xffffffffu, cs[q], 8);
            cs[q] += __shfl_xor_sync(0xffffffffu, cs[q], 16);
          }
          const int pieces = (rows + SUM_ROWS - 1) / SUM_ROWS;
          bool done = pieces == 1;
          if (!done) {
            if (lane < 8 && col < p.m) store8(p.sums + slot * p.m + col, cs);
            __threadfence();
            __syncwarp();
            int before = 0;
            if (lane == 0) before = atomicAdd(p.sum_counts + static_cast<long>(lo) * col_blocks + cb, 1);
            done = __shfl_sync(0xffffffffu, before, 0) == pieces - 1;
            if (done) {
              __threadfence();
              if (lane < 8 && col < p.m) {
#pragma unroll
                for (int q = 0; q < 8; ++q) cs[q] = 0.f;
                for (int i = 0; i < pieces; ++i) {
                  const float4* src = reinterpret_cast<const float4*>(p.sums + (first_slot + i) * p.m + col);
                  const float4 a = __ldcg(src), b = __ldcg(src + 1);
                  cs[0] += a.x; cs[1] += a.y; cs[2] += a.z; cs[3] += a.w;
                  cs[4] += b.x; cs[5] += b.y; cs[6] += b.z; cs[7] += b.w;
                }
              }
            }
          }
          if (done && lane < 8 && col < p.m) store8(p.psum + static_cast<long>(lo) * p.m + col, cs);
        }
      }
      const long elems = static_cast<long>(p.m) * p.n;   // a multiple of 64
      const uint32_t zero[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      for (int g = 0; g < p.num_groups; ++g) {
        if (sh->offs[g + 1] != sh->offs[g]) continue;
        float* dst = p.out + g * elems;
        for (long i = ((static_cast<long>(blockIdx.x) * 2 + side) * 32 + lane) * 8; i < elems; i += static_cast<long>(gridDim.x) * 512) {
          gg::st256(dst + i, zero);
        }
        if (p.psum != nullptr && side == 0 && g % static_cast<int>(gridDim.x) == static_cast<int>(blockIdx.x)) {
          for (int i = lane; i < p.m; i += 32) p.psum[static_cast<long>(g) * p.m + i] = 0.f;
        }
      }
    } else if (KIND == kSplitPlain) {
      // ============================================================ rows past the last expert
      const uint32_t zero[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      const long end = p.rows_cap * p.n;
      for (long i = static_cast<long>(sh->offs[p.num_groups]) * p.n + ((static_cast<long>(blockIdx.x) * 2 + side) * 32 + lane) * 8;
           i < end; i += static_cast<long>(gridDim.x) * 512) {
        gg::st256(p.out + i, zero);
      }
    }
  } else {
    // ============================================================== epilogue (warps 4..11)
    const int part = warp & 3;                       // TMEM lane quarter this warp may read
    const int half = (warp - FIRST_EPI_WARP) >> 2;   // which half of the accumulator columns
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(part * 32) << 16) + half * EPI_COLS;
    int buf = 0;
    uint32_t buf_phase = 0, small_phase = 0;
    bool dead = false;   // a wait ran out: touch nothing else
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (ptx::mbar_wait(bar, parity, abort_flag)) return true;
      if (lane == 0) {
        sh->abort = 1;
        if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_EPILOGUE);
      }
      return false;
    };
    auto release = [&](uint64_t* bar) {
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa(bar, 0));
    };
    while (!dead && walk.next(part_of)) {
      const Tile c = decode(sh, n_tiles, part_of);
      if (KIND == kSplitDAct && ACT != kActNone && part_of.kb0 == 0) {
        const int r = c.m_tile * TILE_M + rank * CTA_M + part * 32 + lane, col = c.n_tile * TILE_N + half * EPI_COLS;
        const float* at = p.pre + (static_cast<long>(c.row_begin) + r) * p.n + col;
        if (r < c.rows && col < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
        if (r < c.rows && col + 32 < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 32));
      }
      ptx::f32x2 acc[EPI_COLS / 2];
#pragma unroll
      for (int j = 0; j < EPI_COLS / 2; ++j) acc[j] = 0ull;
      for (int kb = part_of.kb0; kb < part_of.kb1; ++kb) {
        if (!wait(&sh->main_full[buf], buf_phase)) {
          dead = true;
          break;
        }
        ptx::tc_fence_after_sync();
        uint32_t r0[32], r1[32];
        ptx::tmem_ld_32x32(t_lane + buf * TILE_N, r0);
        ptx::tmem_ld_32x32(t_lane + buf * TILE_N + 32, r1);
        ptx::tmem_ld_wait();
        release(&sh->main_empty[buf]);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          acc[j] = ptx::add2(acc[j], ptx::pack2(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1])));
          acc[16 + j] = ptx::add2(acc[16 + j], ptx::pack2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1])));
        }
        if (++buf == MAIN_BUFS) { buf = 0; buf_phase ^= 1; }
      }
      if (dead || !wait(&sh->small_full, small_phase)) {
        dead = true;
        break;
      }
      small_phase ^= 1;
      ptx::tc_fence_after_sync();
      float v[EPI_COLS];
#pragma unroll
      for (int q = 0; q < 2; ++q) {   // 32 columns at a time: both sums of small products
        uint32_t rm[32], rl[32];
        ptx::tmem_ld_32x32(t_lane + M_COL + q * 32, rm);
        ptx::tmem_ld_32x32(t_lane + L_COL + q * 32, rl);
        ptx::tmem_ld_wait();
        if (q == 1) release(&sh->small_empty);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float a0, a1;
          ptx::unpack2(acc[q * 16 + j], a0, a1);
          const float s0 = join3(a0, __uint_as_float(rm[2 * j]), __uint_as_float(rl[2 * j]));
          const float s1 = join3(a1, __uint_as_float(rm[2 * j + 1]), __uint_as_float(rl[2 * j + 1]));
          v[q * 32 + 2 * j] = fabsf(s0) <= FLT_MAX ? s0 : a0;
          v[q * 32 + 2 * j + 1] = fabsf(s1) <= FLT_MAX ? s1 : a1;
        }
      }
      const int ew = warp - FIRST_EPI_WARP;
      if (part_of.kb0 != 0) {
        // another pair's tile: hand the sum over
        const int slot = (pair * 2 + rank) * NUM_EPI_WARPS + ew;
        float4* dst = reinterpret_cast<float4*>(p.work + static_cast<long>(slot) * WORK_FLOATS) + lane;
#pragma unroll
        for (int j = 0; j < EPI_COLS / 4; ++j) {
          __stcg(dst + j * 32, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) ptx::st_release(p.flags + slot, 1);
        continue;
      }
      for (int q = pair + 1; q <= part_of.last_piece; ++q) {
        const int slot = (q * 2 + rank) * NUM_EPI_WARPS + ew;
        if (!ptx::wait_flag(p.flags + slot, abort_flag, COLLECT_LIMIT_NS)) {
          if (lane == 0) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_COLLECT);
          }
          dead = true;
          break;
        }
        const float4* src = reinterpret_cast<const float4*>(p.work + static_cast<long>(slot) * WORK_FLOATS) + lane;
#pragma unroll
        for (int j = 0; j < EPI_COLS / 4; ++j) {
          const float4 w = __ldcg(src + j * 32);
          v[4 * j] += w.x;
          v[4 * j + 1] += w.y;
          v[4 * j + 2] += w.z;
          v[4 * j + 3] += w.w;
        }
      }
      if (dead) break;
      const int row = c.m_tile * TILE_M + rank * CTA_M + part * 32 + lane;   // in the group
      const int col0 = c.n_tile * TILE_N + half * EPI_COLS;
      const bool row_ok = row < (MODE == kWgrad ? p.m : c.rows);
      const bool pad_ok = KIND != kSplitPlain && row < (c.rows + 63) / 64 * 64;
      const long out_row = (MODE == kWgrad ? static_cast<long>(c.group) * p.m : c.row_begin) + row;
      // 16 columns at a time: a lane has a row of its own, so that each store of a warp touches 32 lines
      // whatever its width, and the widest are the fewest (32 bytes to a plane where the rows allow it).
      // With 16-byte stores and loads behind the stores, 8 experts, 4096 rows, 512 -> 2048 took 131 us with
      // GELU and 115 in its derivative, 104 and 103 so; 16 experts, 8192 rows, 256 -> 1024 110 and 95, 79 and 84.
      // (With three accumulators for h h; with the two there are 106, 116, 82 and 90.)
      float x[16];
      auto load_pre = [&](int col, float (&to)[16]) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t r[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
          if (row_ok && col + 8 * u < p.n) gg::ld256(p.pre + out_row * p.n + col + 8 * u, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) to[8 * u + j] = __uint_as_float(r[j]);
        }
      };
      if (KIND == kSplitDAct && ACT != kActNone) load_pre(col0, x);
#pragma unroll
      for (int q = 0; q < EPI_COLS / 16; ++q) {
        const int col = col0 + q * 16;
        float next[16];   // (the loads of the next columns go ahead of this one's stores)
        if (KIND == kSplitDAct && ACT != kActNone && q + 1 < EPI_COLS / 16) load_pre(col + 16, next);
        if (col < p.n && (row_ok || pad_ok)) {
          uint32_t w[3][8];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float* t = v + q * 16 + u * 8;
            const bool in = col + 8 * u < p.n;
            if (MODE == kRowsNT && KIND != kSplitDAct && p.bias != nullptr && in) {
              float bv[8];
              load8(p.bias + static_cast<long>(c.group) * p.n + col + 8 * u, bv);
#pragma unroll
              for (int j = 0; j < 8; ++j) t[j] += bv[j];
            }
            if (KIND != kSplitDAct && row_ok && in && (KIND == kSplitPlain || p.pre != nullptr)) {
              uint32_t r[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) r[j] = __float_as_uint(t[j]);
              gg::st256((KIND == kSplitPlain ? p.out : p.pre) + out_row * p.n + col + 8 * u, r);
            }
            if (KIND != kSplitPlain) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if (KIND == kSplitAct) t[j] = act32<ACT>(t[j]);
                if (KIND == kSplitDAct) t[j] = act32_bwd<ACT>(t[j], x[8 * u + j]);
                t[j] = row_ok ? t[j] : 0.f;
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) split2(t[2 * j], t[2 * j + 1], w[0][4 * u + j], w[1][4 * u + j], w[2][4 * u + j]);
            }
          }
          if (KIND != kSplitPlain) {
            bf16* dst = p.planes + (c.padded + row) * p.n + col;
#pragma unroll
            for (int pl = 0; pl < 3; ++pl, dst += p.plane_rows * p.n) {
              if ((p.n & 15) == 0) {
                gg::st256(dst, w[pl]);
              } else {
                *reinterpret_cast<uint4*>(dst) = make_uint4(w[pl][0], w[pl][1], w[pl][2], w[pl][3]);
                if (col + 8 < p.n) *reinterpret_cast<uint4*>(dst + 8) = make_uint4(w[pl][4], w[pl][5], w[pl][6], w[pl][7]);
              }
            }
          }
        }
        if (KIND == kSplitDAct && ACT != kActNone && q + 1 < EPI_COLS / 16) {
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = next[j];
        }
      }
      __syncwarp();
    }
  }

  // ---------------------------------------------------------------- tear-down
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

// ------------------------------------------------------------------------------ splitting
constexpr int kSplitThreads = 256;

// Every kernel that splits can zero the flags of GEMMs that follow it.
__device__ __forceinline__ void zero_flags(int* flags, int count) {
  for (int i = blockIdx.x * kSplitThreads + threadIdx.x; i < count; i += gridDim.x * kSplitThreads) flags[i] = 0;
}

// The weights of experts without rows are left out.
__global__ void __launch_bounds__(kSplitThreads)
split_weight_kernel(const float* __restrict__ src, const int* __restrict__ offs, long per_expert, long n, bf16* __restrict__ planes) {
  ptx::chain_begin();
  const long i = (static_cast<long>(blockIdx.x) * kSplitThreads + threadIdx.x) * 8;
  if (i >= n) return;
  const int e = static_cast<int>(i / per_expert);
  if (offs[e] == offs[e + 1]) return;
  float v[8];
  load8(src + i, v);
  store_split8(planes + i, n, v);
}

// 16 padded rows per block.
__global__ void __launch_bounds__(kSplitThreads)
split_rows_kernel(const float* __restrict__ src, const int* __restrict__ offs, int num_groups, long plane_rows, int width,
                  bf16* __restrict__ planes, int* flags, int num_flags) {
  ptx::chain_begin();
  zero_flags(flags, num_flags);
  const int lane = threadIdx.x & 31;
  const long r0 = static_cast<long>(blockIdx.x) * 16;
  int begin = 0, rows = 0;
  long first = 0;
  bool found = false;
  for (int g0 = 0; g0 < num_groups && !found; g0 += 32) {
    const int g = g0 + lane;
    const int lo = g < num_groups ? offs[g] : 0;
    const int cnt = g < num_groups ? offs[g + 1] - lo : 0;
    const long at = split_row(lo, g);
    const unsigned hit = __ballot_sync(0xffffffffu, r0 >= at && r0 < at + (cnt + 63) / 64 * 64);
    if (hit != 0) {
      const int who = __ffs(hit) - 1;
      found = true;
      begin = __shfl_sync(0xffffffffu, lo, who);
      rows = __shfl_sync(0xffffffffu, cnt, who);
      first = __shfl_sync(0xffffffffu, static_cast<int>(r0 - at), who);   // row in the expert
    }
  }
  if (!found) return;
  const int nv = width >> 3;
  for (int it = threadIdx.x; it < 16 * nv; it += kSplitThreads) {
    const int r = it / nv, c = (it - r * nv) * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (first + r < rows) load8(src + (begin + first + r) * width + c, v);
    store_split8(planes + (r0 + r) * width + c, plane_rows * width, v);
  }
}

// Backward of the weighted combine into fp32 rows.  One warp per slot.
__global__ void __launch_bounds__(kSplitThreads)
combine_bwd_f32_kernel(const float* __restrict__ dout, const float* __restrict__ rows, const int64_t* __restrict__ idx,
                       const int* __restrict__ rank, const int* __restrict__ offs, const float* __restrict__ score,
                       long n_slots, int k, int width, float* __restrict__ drows, float* __restrict__ dscore) {
  ptx::chain_begin();
  const int lane = threadIdx.x & 31;
  const long s = static_cast<long>(blockIdx.x) * (kSplitThreads / 32) + (threadIdx.x >> 5);
  if (s >= n_slots) return;
  const int rk = rank[s];
  if (rk < 0) {
    if (lane == 0) dscore[s] = 0.f;
    return;
  }
  const long row = static_cast<long>(offs[idx[s]]) + rk;
  const float w = score[s];
  float dot = 0.f;
  for (int i = lane; i < (width >> 3); i += 32) {
    float g[8], y[8];
    load8(dout + s / k * width + i * 8, g);
    load8(rows + row * width + i * 8, y);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      dot += g[q] * y[q];
      g[q] *= w;
    }
    store8(drows + row * width + i * 8, g);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (lane == 0) dscore[s] = dot;
}

// One warp per slot; the blocks behind those of the slots write the zero rows of one expert each.
// BWD: the rows are scaled by their slot's score, whose gradient is formed on the way.
template <bool BWD>
__global__ void __launch_bounds__(kSplitThreads)
split_scatter_kernel(const float* __restrict__ src, const float* __restrict__ rows, const int64_t* __restrict__ idx,
                     const int* __restrict__ rank, const int* __restrict__ offs, const float* __restrict__ score,
                     int num_groups, long n_slots, int k, int width, long plane_rows, int slot_blocks,
                     bf16* __restrict__ planes, float* __restrict__ dscore, int* flags, int num_flags) {
  ptx::chain_begin();
  zero_flags(flags, num_flags);
  const int lane = threadIdx.x & 31;
  const int nv = width >> 3;
  const long plane = plane_rows * width;
  if (static_cast<int>(blockIdx.x) >= slot_blocks) {
    const int g = static_cast<int>(blockIdx.x) - slot_blocks;
    const int lo = offs[g], cnt = offs[g + 1] - lo;
    const int pad = (cnt + 63) / 64 * 64 - cnt;
    const float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int it = threadIdx.x; it < pad * nv; it += kSplitThreads) {
      const int r = it / nv, c = (it - r * nv) * 8;
      store_split8(planes + (split_row(lo, g) + cnt + r) * width + c, plane, zero);
    }
    return;
  }
  const long s = static_cast<long>(blockIdx.x) * (kSplitThreads / 32) + (threadIdx.x >> 5);
  if (s >= n_slots) return;
  const int rk = rank[s];   // negative for dropped slots and for ids that name no expert
  if (rk < 0) {
    if (BWD && lane == 0) dscore[s] = 0.f;
    return;
  }
  const long e = idx[s];
  const int lo = offs[e];
  const float* in = src + s / k * width;
  bf16* out = planes + (split_row(lo, e) + rk) * width;
  if (!BWD) {
    for (int i = lane; i < nv; i += 32) {
      float v[8];
      load8(in + i * 8, v);
      store_split8(out + i * 8, plane, v);
    }
  } else {
    const float* y = rows + (static_cast<long>(lo) + rk) * width;
    const float w = score[s];
    float dot = 0.f;
    for (int i = lane; i < nv; i += 32) {
      float g[8], yv[8];
      load8(in + i * 8, g);
      load8(y + i * 8, yv);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        dot += g[q] * yv[q];
        g[q] *= w;
      }
      store_split8(out + i * 8, plane, g);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) dscore[s] = dot;
  }
}

// One warp per token.
__global__ void __launch_bounds__(kSplitThreads)
combine_f32_kernel(const float* __restrict__ rows, const int64_t* __restrict__ idx, const int* __restrict__ rank,
                   const int* __restrict__ offs, const float* __restrict__ weight, long n_tokens, int k,
                   int width, float* __restrict__ out) {
  ptx::chain_begin();
  const int lane = threadIdx.x & 31;
  const long t = static_cast<long>(blockIdx.x) * (kSplitThreads / 32) + (threadIdx.x >> 5);
  if (t >= n_tokens) return;
  for (int i = lane; i < (width >> 3); i += 32) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < k; ++j) {
      const long s = t * k + j;
      const int rk = rank[s];
      if (rk < 0) continue;
      const float w = weight != nullptr ? weight[s] : 1.f;
      float v[8];
      load8(rows + (static_cast<long>(offs[idx[s]]) + rk) * width + i * 8, v);
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] += w * v[q];
    }
    store8(out + t * width + i * 8, acc);
  }
}

// ------------------------------------------------------------------------------ launch
template <int MODE, int KIND, int ACT>
cudaError_t launch_one(const CUtensorMap& ta, const CUtensorMap& tb, const Params& p, int grid, cudaStream_t stream) {
  static std::mutex mu;   // the shared-memory attribute is per device
  static uint64_t configured = 0;
  auto kernel = split_gemm_kernel<MODE, KIND, ACT>;
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
  return launch_chained(kernel, dim3(grid), dim3(NUM_THREADS), SMEM_BYTES, stream, ta, tb, p);
}

template <int MODE, int KIND>
cudaError_t launch_act(int act, const CUtensorMap& ta, const CUtensorMap& tb, const Params& p, int grid, cudaStream_t stream) {
  switch (act) {
    case kActRelu: return launch_one<MODE, KIND, kActRelu>(ta, tb, p, grid, stream);
    case kActGelu: return launch_one<MODE, KIND, kActGelu>(ta, tb, p, grid, stream);
    case kActGeluTanh: return launch_one<MODE, KIND, kActGeluTanh>(ta, tb, p, grid, stream);
    default: return launch_one<MODE, KIND, kActNone>(ta, tb, p, grid, stream);
  }
}

unsigned blocks_of(long items, long per) { return static_cast<unsigned>((items + per - 1) / per); }

}  // namespace

long split_work_floats(int num_sms) { return static_cast<long>(num_sms) * NUM_EPI_WARPS * WORK_FLOATS; }
int split_num_flags(int num_sms) { return num_sms * NUM_EPI_WARPS; }
long split_sum_floats(long rows_cap, int num_groups, int m) { return (sum_slot(rows_cap, num_groups) + 1) * m; }
int split_num_counts(int num_groups, int m) { return num_groups * ((m + 63) / 64); }

bool split_gemm_supported(int mode, int m, int n, int k, int num_groups, long rows_cap) {
  const int inner = mode == kWgrad ? m : k;
  return num_groups >= 1 && num_groups <= MAX_GROUPS && n >= 16 && n % 8 == 0 && inner >= 16 && inner % 8 == 0 &&
         rows_cap > 0 && 3 * split_rows_cap(rows_cap, num_groups) <= INT32_MAX &&
         3L * num_groups * (mode == kRowsNN ? 1 : n) <= INT32_MAX;
}

cudaError_t launch_split_gemm(const SplitGemmArgs& a) {
  if (!split_gemm_supported(a.mode, a.m, a.n, a.k, a.num_groups, a.rows_cap)) return cudaErrorInvalidValue;
  const uint64_t rp = split_rows_cap(a.rows_cap, a.num_groups), groups = a.num_groups;
  CUtensorMap ta, tb;
  bool ok;
  if (a.mode == kWgrad) {
    ok = make_map_2d(&ta, kBF16, a.a, a.m, 3 * rp, 64, BK) && make_map_2d(&tb, kBF16, a.b, a.n, 3 * rp, 64, BK);
  } else {
    ok = make_map_2d(&ta, kBF16, a.a, a.k, 3 * rp, BK, CTA_M) &&
         (a.mode == kRowsNT ? make_map_2d(&tb, kBF16, a.b, a.k, 3 * groups * a.n, BK, CTA_N)
                            : make_map_3d(&tb, kBF16, a.b, a.n, a.k, 3 * groups, 64, BK));
  }
  if (!ok) return cudaErrorInvalidValue;
  Params p;
  p.num_groups = a.num_groups;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.rows_cap = a.rows_cap;
  p.plane_rows = static_cast<long>(rp);
  p.offs = a.offs;
  p.bias = a.bias;
  p.out = a.out;
  p.planes = static_cast<bf16*>(a.planes);
  p.pre = a.pre;
  p.psrc = static_cast<const bf16*>(a.a);
  p.psum = a.psum;
  p.work = a.work;
  p.flags = a.flags;
  p.sums = a.sums;
  p.sum_counts = a.sum_counts;
  if (a.psum != nullptr && (a.sums == nullptr || a.sum_counts == nullptr)) return cudaErrorInvalidValue;
  p.status = a.status;
  const int grid = (a.num_sms > 1 ? a.num_sms : 148) & ~1;
  if (a.mode == kWgrad) return launch_one<kWgrad, kSplitPlain, kActNone>(ta, tb, p, grid, a.stream);
  if (a.mode == kRowsNT) {
    return a.kind == kSplitAct ? launch_act<kRowsNT, kSplitAct>(a.act, ta, tb, p, grid, a.stream)
                               : launch_one<kRowsNT, kSplitPlain, kActNone>(ta, tb, p, grid, a.stream);
  }
  return a.kind == kSplitDAct ? launch_act<kRowsNN, kSplitDAct>(a.act, ta, tb, p, grid, a.stream)
                              : launch_one<kRowsNN, kSplitPlain, kActNone>(ta, tb, p, grid, a.stream);
}

cudaError_t launch_split_weight(const float* src, const int* offs, int num_groups, long per_expert, void* planes,
                                cudaStream_t stream) {
  const long n = num_groups * per_expert;
  return launch_chained(split_weight_kernel, dim3(blocks_of(n, kSplitThreads * 8)), dim3(kSplitThreads), 0, stream, src, offs,
                        per_expert, n, static_cast<bf16*>(planes));
}

cudaError_t launch_split_rows(const float* src, const int* offs, int num_groups, long rows_cap, int width, void* planes,
                              int* flags, int num_flags, cudaStream_t stream) {
  const long rp = split_rows_cap(rows_cap, num_groups);
  return launch_chained(split_rows_kernel, dim3(blocks_of(rp, 16)), dim3(kSplitThreads), 0, stream, src, offs, num_groups, rp,
                        width, static_cast<bf16*>(planes), flags, num_flags);
}

cudaError_t launch_split_scatter(const float* src, const int64_t* idx, const int* rank, const int* offs, int num_groups,
                                 long n_slots, int k, int width, void* planes, int* flags, int num_flags,
                                 cudaStream_t stream) {
  const unsigned blocks = blocks_of(n_slots, kSplitThreads / 32);
  return launch_chained(split_scatter_kernel<false>, dim3(blocks + num_groups), dim3(kSplitThreads), 0, stream, src,
                        static_cast<const float*>(nullptr), idx, rank, offs, static_cast<const float*>(nullptr), num_groups,
                        n_slots, k, width, split_rows_cap(n_slots, num_groups), static_cast<int>(blocks),
                        static_cast<bf16*>(planes), static_cast<float*>(nullptr), flags, num_flags);
}

cudaError_t launch_split_combine_bwd(const float* dout, const float* rows, const int64_t* idx, const int* rank,
                                     const int* offs, const float* score, int num_groups, long n_slots, int k, int width,
                                     void* planes, float* dscore, int* flags, int num_flags, cudaStream_t stream) {
  const unsigned blocks = blocks_of(n_slots, kSplitThreads / 32);
  return launch_chained(split_scatter_kernel<true>, dim3(blocks + num_groups), dim3(kSplitThreads), 0, stream, dout, rows,
                        idx, rank, offs, score, num_groups, n_slots, k, width, split_rows_cap(n_slots, num_groups),
                        static_cast<int>(blocks), static_cast<bf16*>(planes), dscore, flags, num_flags);
}

cudaError_t launch_combine_f32(const float* rows, const int64_t* idx, const int* rank, const int* offs,
                               const float* weight, long n_tokens, int k, int width, float* out, cudaStream_t stream) {
  if (n_tokens == 0) return cudaSuccess;
  return launch_chained(combine_f32_kernel, dim3(blocks_of(n_tokens, kSplitThreads / 32)), dim3(kSplitThreads), 0, stream, rows,
                        idx, rank, offs, weight, n_tokens, k, width, out);
}

cudaError_t launch_combine_bwd_f32(const float* dout, const float* rows, const int64_t* idx, const int* rank,
                                   const int* offs, const float* score, long n_slots, int k, int width, float* drows,
                                   float* dscore, cudaStream_t stream) {
  if (n_slots == 0) return cudaSuccess;
  return launch_chained(combine_bwd_f32_kernel, dim3(blocks_of(n_slots, kSplitThreads / 32)), dim3(kSplitThreads), 0, stream,
                        dout, rows, idx, rank, offs, score, n_slots, k, width, drows, dscore);
}

}  // namespace fmoe
