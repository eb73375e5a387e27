// Grouped GEMM on CTA pairs, row modes (forward and input gradient): the token rows are the N side of
// the MMA.
//
// With tiles of 256 token rows, as the weight gradient's kernel has them and this one's predecessor had, an
// expert with 130 rows costs as much as one with 256, the second CTA has next to nothing to store, and half
// of what is loaded are other experts' rows.  Here a tile is 256 output columns (rows of the weights, M) by
// as many token rows as the expert has left, in steps of 64 and at most 256 (N, chosen tile by tile in the
// instruction descriptor), so that both the MMAs and the loads go with the rows there are and the epilogue is
// shared evenly by the two CTAs.  What bounds it: with up to a hundred rows per expert the weights (64
// experts, 64 rows each, 1024 -> 4096, no activation: 100 us, 5.4 TB/s); with many rows the tensor cores
// (8192 rows, 2 experts, 1024 <-> 4096: 53 and 51 us, 1280 to 1340 TFLOP/s) and, with few K blocks, the
// epilogue.  Against 256-row tiles: see the rule in grouped_gemm.cu.
//
// The accumulators come out transposed: a TMEM lane is an output column, a TMEM column a token row.  The
// epilogue loads them as 8 x 8 fragments (tcgen05.ld 16x256b) and transposes them on the way to shared
// memory (stmatrix.trans); 32 rows x 64 bytes leave by TMA.  The saved pre-activation is the same
// tile-blocked buffer as elsewhere.
//
// Roles of a CTA (384 threads), persistent over the tiles of its pair: warp 0 loads, warp 1 of CTA 0
// issues the MMAs, warps 4-11 finish 32 output columns each, four warps every other 32 token rows.
#pragma once
#include "pair_gemm_kernel.cuh"

namespace fmoe {
namespace slim {

using gg::Cvt;
using pg::PAIRS;

constexpr int TILE_N = 256;                  // output columns per tile
constexpr int CTA_N = TILE_N / 2;
constexpr int MAX_ROWS = 256;                // token rows per tile
constexpr int ROW_STEP = 64;                 // ... in steps of
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int STAGES = 5;
constexpr int W_BYTES = CTA_N * BK * 2;
constexpr int X_BYTES = MAX_ROWS / 2 * BK * 2;
constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
constexpr int BOX_BYTES = 64 * BK * 2;
constexpr int HALF_STEP = ROW_STEP / 2;      // a CTA loads half of the tile's token rows: 32, 64, 96 or 128
constexpr int HALF_SIZES = MAX_ROWS / ROW_STEP;
constexpr int MAX_GROUPS = gg::MAX_GROUPS;
constexpr int NUM_EPI_WARPS = 8;
constexpr int FIRST_EPI_WARP = 4;
constexpr int NUM_THREADS = (FIRST_EPI_WARP + NUM_EPI_WARPS) * 32;
constexpr int PATCH_BYTES = 32 * 64;         // 32 token rows x 32 columns
constexpr int PATCHES = 3;                   // per warp: two for results in turn, one for the pre-activation
constexpr int TMEM_COLS = 512;

struct Shared {
  uint64_t full[STAGES];        // CTA 0's counts: one arrival and the bytes of each CTA
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];       // CTA 0's counts: every epilogue warp of both CTAs
  uint32_t tmem_base;
  int abort;
  int offs[MAX_GROUPS + 1];
  int tiles[MAX_GROUPS + 1];    // exclusive prefixes of the tiles and of the 128-row blocks of the pre-activation
  int blocks[MAX_GROUPS + 1];
};
constexpr int PATCH_OFF = STAGES * STAGE_BYTES;
constexpr int AUX_OFF = PATCH_OFF + NUM_EPI_WARPS * PATCHES * PATCH_BYTES;
constexpr int SMEM_BYTES = AUX_OFF + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory");

// A copy per K block and operand, whatever the tile's size: with boxes of 32 token rows the loading
// thread issued up to six, and 8 experts with 128 rows, 4096 -> 1024 took 30 us instead of 26.
struct Maps {
  CUtensorMap w;               // weights
  CUtensorMap x[HALF_SIZES];   // token rows, boxes of 32, 64, 96 and 128
  CUtensorMap c;               // output
};

struct Params {
  int num_groups;
  int n, k;
  int w_blocks;          // input gradient: `w` counts blocks of 64 columns, two to a box
  const int* offs;       // null: `one_group` instead
  int one_group[2];
  void* out;
  void* pre_out;
  const void* bias;
  const void* aux;
  int* status;
};

struct Tile {
  int group, n_tile;
  int row0, valid;       // first token row and rows of the tile
  int first;             // its first row in the expert
  int mma_n;             // rows the MMA takes
};

__device__ __forceinline__ Tile decode(const Shared* sh, int n_tiles, int tile, int& hint) {
  int g = hint;
  while (sh->tiles[g + 1] <= tile) ++g;
  hint = g;
  const int local = tile - sh->tiles[g];
  const int m = local / n_tiles;
  Tile t;
  t.group = g;
  t.n_tile = local - m * n_tiles;
  t.first = m * MAX_ROWS;
  t.row0 = sh->offs[g] + t.first;
  t.valid = min(MAX_ROWS, sh->offs[g + 1] - t.row0);
  t.mma_n = (t.valid + ROW_STEP - 1) / ROW_STEP * ROW_STEP;
  return t;
}

// 16-byte piece `c` (0..3) of patch row `row`; swizzled as a tensor map with 64-byte swizzle is.
__device__ __forceinline__ uint32_t patch_piece(uint32_t patch, int row, int c) {
  return patch + row * 64 + ((c ^ ((row >> 1) & 3)) << 4);
}

// A chunk of 32 columns x 32 token rows as fragments: frag[s][4 j + 2 i + v] is column 16 s + 8 i + lane / 4,
// token row 8 j + 2 (lane % 4) + v.
struct Fragments {
  uint32_t r[2][16];
};

// Packed to 16 bits and transposed into the patch: rows of 32 columns.
template <typename T> __device__ __forceinline__ void put_chunk(uint32_t patch, int lane, const ptx::f32x2 (&v)[2][8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t w[4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float a, b;
        ptx::unpack2(v[s][2 * j + i], a, b);
        w[2 * s + i] = Cvt<T>::pack(a, b);
      }
    }
    ptx::stmatrix_x4_trans(patch_piece(patch, 8 * j + (lane & 7), lane >> 3), w);
  }
}

template <int MODE, typename T, int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
slim_gemm_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + AUX_OFF);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(ptx::cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x) >> 1;
  const int num_pairs = static_cast<int>(gridDim.x) >> 1;
  const int n_tiles = (p.n + TILE_N - 1) / TILE_N;
  const int num_kb = p.k / BK;
  const volatile int* abort_flag = &sh->abort;

  // ---------------------------------------------------------------- set-up
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&sh->full[s], 2);
      ptx::mbar_init(&sh->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&sh->tmem_full[a], 1);
      ptx::mbar_init(&sh->tmem_empty[a], 2 * NUM_EPI_WARPS);
    }
    sh->abort = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&maps.w);
    for (int i = 0; i < HALF_SIZES; ++i) ptx::prefetch_tmap(&maps.x[i]);
    ptx::prefetch_tmap(&maps.c);
  }
  if (warp == 1) ptx::tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
  ptx::chain_begin();   // nothing an earlier kernel writes is read above
  if (warp == 2) {
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
      int t = (rows + MAX_ROWS - 1) / MAX_ROWS * n_tiles;
      int b = (rows + 127) / 128;
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
        const int n0 = c.n_tile * TILE_N + rank * CTA_N;
        const int half = c.mma_n / 2;
        const int x0 = c.row0 + rank * half;
        const CUtensorMap* tm_x = &maps.x[half / HALF_STEP - 1];
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          uint8_t* sw = smem + stage * STAGE_BYTES;
          uint8_t* sx = sw + W_BYTES;
          const uint32_t bar = ptx::mapa(&sh->full[stage], 0);
          ptx::mbar_arrive_expect_tx_cluster(bar, W_BYTES + half * (BK * 2));
          if (MODE == kRowsNT) {
            ptx::tma_load_2d_pair(sw, &maps.w, bar, kb * BK, c.group * p.n + n0);
          } else if (p.w_blocks) {
            ptx::tma_load_3d_pair(sw, &maps.w, bar, 0, c.group * p.k + kb * BK, n0 / 64);
          } else {
            ptx::tma_load_2d_pair(sw, &maps.w, bar, n0, c.group * p.k + kb * BK);
            ptx::tma_load_2d_pair(sw + BOX_BYTES, &maps.w, bar, n0 + 64, c.group * p.k + kb * BK);
          }
          ptx::tma_load_2d_pair(sx, tm_x, bar, kb * BK, x0);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ============================================================== MMA issuer (CTA 0)
    if (rank == 0 && lane == 0) {
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      int stage = 0;
      uint32_t phase = 0;
      int iter = 0;
      bool ok = true;
      for (int tile = pair; tile < total && ok; tile += num_pairs, ++iter) {
        const Tile c = decode(sh, n_tiles, tile, group);
        const uint32_t idesc = ptx::make_idesc(kBf16, MODE == kRowsNN, false, TILE_N, c.mma_n);
        const int acc = iter & 1;
        if (!ptx::mbar_wait(&sh->tmem_empty[acc], ((iter >> 1) & 1) ^ 1, abort_flag)) {
          sh->abort = 1;
          if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * MAX_ROWS;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&sh->full[stage], phase, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sw = ptx::smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sx = sw + W_BYTES;
#pragma unroll
          for (int k16 = 0; k16 < BK / UMMA_K; ++k16) {
            const uint64_t w_desc = MODE == kRowsNN ? ptx::make_smem_desc_sw128(sw + k16 * (UMMA_K * 128), BOX_BYTES, 1024)
                                                    : ptx::make_smem_desc_sw128(sw + k16 * (UMMA_K * 2), 16, 1024);
            const uint64_t x_desc = ptx::make_smem_desc_sw128(sx + k16 * (UMMA_K * 2), 16, 1024);
            ptx::umma_f16_pair(d_tmem, w_desc, x_desc, idesc, (kb | k16) != 0 ? 1u : 0u);
          }
          ptx::umma_commit_pair(&sh->empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        ptx::umma_commit_pair(&sh->tmem_full[acc]);
      }
    }
  } else if (warp >= FIRST_EPI_WARP) {
    // ============================================================== epilogue (warps 4..11)
    constexpr bool kDAct = MODE == kRowsNN && ACT != kActNone;
    const int ew = warp - FIRST_EPI_WARP;
    const int part = warp & 3;       // TMEM lane quarter this warp may read: its 32 output columns
    const int odd = ew >> 2;         // which chunks of 32 token rows
    const uint32_t patch = ptx::smem_u32(smem + PATCH_OFF + ew * PATCHES * PATCH_BYTES);
    const uint32_t side = patch + 2 * PATCH_BYTES;
    const bool has_bias = MODE == kRowsNT && p.bias != nullptr;
    int iter = 0, buf = 0;
    for (int tile = pair; tile < total; tile += num_pairs, ++iter) {
      const Tile c = decode(sh, n_tiles, tile, group);
      const int acc = iter & 1;
      const int n0 = c.n_tile * TILE_N + rank * CTA_N + part * 32;
      const bool cols = n0 < p.n;    // n is a multiple of 32
      const int chunks = cols ? (c.valid + 31) / 32 : 0;
      // this lane's bias values: columns 16 s + 8 i + lane / 4
      float bias[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
      if (has_bias && cols) {
        const T* b = static_cast<const T*>(p.bias) + static_cast<long>(c.group) * p.n + n0 + (lane >> 2);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
#pragma unroll
          for (int i = 0; i < 2; ++i) bias[s][i] = Cvt<T>::to_f(b[16 * s + 8 * i]);
        }
      }
      const uint8_t* pre_base = static_cast<const uint8_t*>(MODE == kRowsNN ? p.aux : p.pre_out);
      const bool with_pre = ACT != kActNone && pre_base != nullptr;
      // a chunk of the tile-blocked pre-activation
      auto pre_chunk = [&](const Tile& t, int chunk) {
        const int row = t.first + chunk * 32;
        const long blk = (static_cast<long>(sh->blocks[t.group]) + row / 128) * n_tiles + t.n_tile;
        return const_cast<uint8_t*>(pre_base) + blk * gg::PRE_TILE_BYTES +
               ((rank * 4 + (row % 128) / 32) * gg::CHUNKS_PER_WARP + part) * gg::PRE_CHUNK_BYTES;
      };
      uint4 pre[4];
      auto load_pre = [&](int chunk) {
        const uint8_t* src = pre_chunk(c, chunk) + lane * 16;
#pragma unroll
        for (int q = 0; q < 4; ++q) pre[q] = __ldg(reinterpret_cast<const uint4*>(src + q * 512));
      };
      if (kDAct) {
        // it does not depend on the accumulator: fetch the first chunk before the wait, and pull those
        // of the next tile (2 KB each) into the L2
        if (odd < chunks) load_pre(odd);
        if (tile + num_pairs < total) {
          int ahead = group;
          const Tile next = decode(sh, n_tiles, tile + num_pairs, ahead);
          const bool there = next.n_tile * TILE_N + rank * CTA_N + part * 32 < p.n;
          for (int chunk = odd + 2 * (lane >> 4); there && chunk * 32 < next.valid; chunk += 4) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(pre_chunk(next, chunk) + (lane & 15) * 128));
          }
        }
      }
      if (!ptx::mbar_wait(&sh->tmem_full[acc], (iter >> 1) & 1, abort_flag)) {
        if (lane == 0) {
          sh->abort = 1;
          if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_EPILOGUE);
        }
        break;
      }
      ptx::tc_fence_after_sync();
      bool released = false;
      auto release = [&]() {
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa(&sh->tmem_empty[acc], 0));
        released = true;
      };
#pragma unroll 1
      for (int chunk = odd; chunk < chunks; chunk += 2) {
        Fragments f;
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(part * 32) << 16) + acc * MAX_ROWS + chunk * 32;
        ptx::tmem_ld_16x256_x4(t_addr, f.r[0]);
        ptx::tmem_ld_16x256_x4(t_addr + (16u << 16), f.r[1]);
        ptx::tmem_ld_wait();
        if (chunk + 2 >= chunks) release();
        // the last copy but one has read the patch whose turn it is
        const uint32_t out_patch = patch + buf * PATCH_BYTES;
        if (lane == 0) ptx::bulk_wait_read<1>();
        __syncwarp();
        ptx::f32x2 v[2][8];   // pairs of token rows: [s][2 j + i]
#pragma unroll
        for (int s = 0; s < 2; ++s) {
#pragma unroll
          for (int q = 0; q < 8; ++q) v[s][q] = ptx::pack2(__uint_as_float(f.r[s][2 * q]), __uint_as_float(f.r[s][2 * q + 1]));
        }
        if (kDAct) {
#pragma unroll
          for (int q = 0; q < 4; ++q) ptx::st_shared_v4(patch_piece(side, lane, q), pre[q]);
          __syncwarp();
          if (chunk + 2 < chunks) load_pre(chunk + 2);
          ptx::f32x2 x[2][8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w[4];
            ptx::ldmatrix_x4_trans(w, patch_piece(side, 8 * j + (lane & 7), lane >> 3));
#pragma unroll
            for (int s = 0; s < 2; ++s) {
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                float a, b;
                Cvt<T>::unpack(w[2 * s + i], a, b);
                x[s][2 * j + i] = ptx::pack2(a, b);
              }
            }
          }
          pg::act_grad_pairs<ACT>(x[0], v[0]);
          pg::act_grad_pairs<ACT>(x[1], v[1]);
        } else {
          if (has_bias) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
#pragma unroll
              for (int q = 0; q < 8; ++q) v[s][q] = ptx::add2(v[s][q], ptx::pack2(bias[s][q & 1], bias[s][q & 1]));
            }
          }
          if (ACT != kActNone) {
            if (with_pre) {
              put_chunk<T>(side, lane, v);
              __syncwarp();
              uint8_t* dst = pre_chunk(c, chunk) + lane * 16;
#pragma unroll
              for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(dst + q * 512) = ptx::ld_shared_v4(patch_piece(side, lane, q));
            }
            pg::act_pairs<ACT>(v[0]);
            pg::act_pairs<ACT>(v[1]);
          }
        }
        put_chunk<T>(out_patch, lane, v);
        const int rows = c.valid - chunk * 32;
        if (rows >= 32) {
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_3d_at(&maps.c, out_patch, n0, c.row0 + chunk * 32, 0);
            ptx::bulk_commit();
          }
          buf ^= 1;
        } else {
          // the expert's last rows, 4 lanes each
          __syncwarp();
          uint8_t* dst = static_cast<uint8_t*>(p.out) + (static_cast<long>(c.row0 + chunk * 32) * p.n + n0) * 2;
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int row = it * 8 + (lane >> 2);
            if (row < rows) {
              *reinterpret_cast<uint4*>(dst + static_cast<long>(row) * p.n * 2 + (lane & 3) * 16) =
                  ptx::ld_shared_v4(patch_piece(out_patch, row, lane & 3));
            }
          }
          __syncwarp();
        }
      }
      if (!released) release();
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
cudaError_t launch_one(const Maps& m, const Params& p, int grid, cudaStream_t stream) {
  static std::mutex mu;   // the shared-memory attribute is per device
  static uint64_t configured = 0;
  auto kernel = slim_gemm_kernel<MODE, T, ACT>;
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
  return launch_chained(kernel, dim3(grid), dim3(NUM_THREADS), SMEM_BYTES, stream, m, p);
}

template <int MODE, typename T>
cudaError_t launch_act(int act, const Maps& m, const Params& p, int grid, cudaStream_t stream) {
  switch (act) {
    case kActRelu: return launch_one<MODE, T, kActRelu>(m, p, grid, stream);
    case kActGelu: return launch_one<MODE, T, kActGelu>(m, p, grid, stream);
    case kActGeluTanh: return launch_one<MODE, T, kActGeluTanh>(m, p, grid, stream);
    default: return launch_one<MODE, T, kActNone>(m, p, grid, stream);
  }
}

// One translation unit per element type instantiates this.
template <typename T>
cudaError_t launch_for_type(int mode, int act, const Maps& m, const Params& p, int grid, cudaStream_t stream) {
  return mode == kRowsNT ? launch_act<kRowsNT, T>(act, m, p, grid, stream) : launch_act<kRowsNN, T>(act, m, p, grid, stream);
}

cudaError_t launch_bf16(int mode, int act, const Maps& m, const Params& p, int grid, cudaStream_t stream);
cudaError_t launch_f16(int mode, int act, const Maps& m, const Params& p, int grid, cudaStream_t stream);

}  // namespace slim
}  // namespace fmoe
