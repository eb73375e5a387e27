// Grouped GEMM for a handful of rows per expert (decoding): out[rows_e, n] = act(x W_e^T + b_e).
//
// All there is to do is to read the weights once.  The product is computed transposed: 128 rows of
// W_e are the M side of the MMA and up to 32 token rows its N side, so that a stage of the ring
// holds 16 KB of weights and 4 KB of rows where a 128 x 256 tile loads 128 rows of x for every
// tile, most of them other experts', and a tile is a quarter of the work: 64 experts, 128 rows,
// 4096 -> 1024 are 440 tiles for 148 SMs where the wide tiles are 222 (1.5 waves).  Ten stages
// keep 200 KB per SM on their way.  Measured there: 74 us per launch for 445 MB of weights in use
// (6.0 TB/s); with fewer tiles than SMs (8 experts, 4096 -> 1024: 56 tiles, 23 us) what one SM can
// load bounds it.
//
// Roles of a CTA (192 threads, persistent over tiles): warp 0 loads (TMA), warp 1 issues the MMAs
// and owns the TMEM, warps 2-5 finish 32 output columns x 32 rows each: lane = output column.
#include "grouped_gemm_kernel.cuh"
#include "launch.cuh"
#include "narrow_gemm.cuh"

namespace fmoe {
namespace ng {
namespace {

using gg::Cvt;

constexpr int UMMA_K = 16;
constexpr int STAGES = 10;
constexpr int W_BYTES = TILE_N * BK * 2;
constexpr int X_BYTES = TILE_ROWS * BK * 2;
constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
constexpr int NUM_THREADS = 192;
constexpr int TMEM_COLS = 2 * TILE_ROWS;

struct Shared {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort;
  int offs[gg::MAX_GROUPS + 1];
  int tiles[gg::MAX_GROUPS + 1];
};
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + static_cast<int>(sizeof(Shared)) + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory");

struct Tile {
  int group, row0, valid, n0;   // first row, rows (at most 32), first output column
};

__device__ __forceinline__ Tile decode(const Shared* sh, int num_groups, int n_tiles, int tile) {
  int lo = 0, hi = num_groups;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sh->tiles[mid] <= tile) lo = mid; else hi = mid;
  }
  const int local = tile - sh->tiles[lo];
  const int r = local / n_tiles;
  Tile t;
  t.group = lo;
  t.n0 = (local - r * n_tiles) * TILE_N;
  t.row0 = sh->offs[lo] + r * TILE_ROWS;
  t.valid = min(TILE_ROWS, sh->offs[lo + 1] - t.row0);
  return t;
}

template <typename T, int ACT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
narrow_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                   const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_tiles = (p.n + TILE_N - 1) / TILE_N;
  const int num_kb = p.k / BK;
  const volatile int* abort_flag = &sh->abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&sh->full[s], 1);
      ptx::mbar_init(&sh->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&sh->tmem_full[a], 1);
      ptx::mbar_init(&sh->tmem_empty[a], 4);
    }
    sh->abort = 0;
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&tm_w);
    ptx::prefetch_tmap(&tm_x);
  }
  if (warp == 1) {
    ptx::tmem_alloc(&sh->tmem_base, TMEM_COLS);
    ptx::tmem_relinquish();
  }
  ptx::chain_begin();   // nothing an earlier kernel writes is read above
  if (warp == 2) {
    const int* offs = p.offs != nullptr ? p.offs : p.one_group;
    int run = 0;
    if (lane == 0) {
      sh->tiles[0] = 0;
      sh->offs[0] = offs[0];
    }
    for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
      const int g = g0 + lane;
      int end = 0, t = 0;
      if (g < p.num_groups) {
        end = offs[g + 1];
        t = (end - offs[g] + TILE_ROWS - 1) / TILE_ROWS * n_tiles;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += up;
      }
      if (g < p.num_groups) {
        sh->offs[g + 1] = end;
        sh->tiles[g + 1] = run + t;
      }
      run += __shfl_sync(0xffffffffu, t, 31);
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = sh->tmem_base;
  const int total = sh->tiles[p.num_groups];

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        const Tile c = decode(sh, p.num_groups, n_tiles, tile);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          uint8_t* sw = smem + stage * STAGE_BYTES;
          ptx::mbar_arrive_expect_tx(&sh->full[stage], STAGE_BYTES);
          ptx::tma_load_2d(sw, &tm_w, &sh->full[stage], kb * BK, c.group * p.n + c.n0);
          ptx::tma_load_2d(sw + W_BYTES, &tm_x, &sh->full[stage], kb * BK, c.row0);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc =
          ptx::make_idesc(std::is_same<T, __nv_bfloat16>::value, false, false, TILE_N, TILE_ROWS);
      int stage = 0;
      uint32_t phase = 0;
      int iter = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x, ++iter) {
        const int acc = iter & 1;
        if (!ptx::mbar_wait(&sh->tmem_empty[acc], ((iter >> 1) & 1) ^ 1, abort_flag)) {
          sh->abort = 1;
          if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
          break;
        }
        ptx::tc_fence_after_sync();
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&sh->full[stage], phase, abort_flag)) {
            sh->abort = 1;
            if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_MMA);
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sw = ptx::smem_u32(smem + stage * STAGE_BYTES);
#pragma unroll
          for (int k16 = 0; k16 < BK / UMMA_K; ++k16) {
            ptx::umma_f16(tmem_base + acc * TILE_ROWS, ptx::make_smem_desc_sw128(sw + k16 * (UMMA_K * 2), 16, 1024),
                          ptx::make_smem_desc_sw128(sw + W_BYTES + k16 * (UMMA_K * 2), 16, 1024), idesc,
                          (kb | k16) != 0 ? 1u : 0u);
          }
          ptx::umma_commit(&sh->empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        ptx::umma_commit(&sh->tmem_full[acc]);
      }
    }
  } else {
    const int part = warp & 3;   // TMEM lane quarter this warp may read
    int iter = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++iter) {
      const Tile c = decode(sh, p.num_groups, n_tiles, tile);
      const int acc = iter & 1;
      const int col = c.n0 + part * 32 + lane;
      const bool on = col < p.n;
      float bias = 0.f;
      if (on && p.bias != nullptr) bias = Cvt<T>::to_f(static_cast<const T*>(p.bias)[static_cast<long>(c.group) * p.n + col]);
      if (!ptx::mbar_wait(&sh->tmem_full[acc], (iter >> 1) & 1, abort_flag)) {
        if (lane == 0) {
          sh->abort = 1;
          if (p.status != nullptr) record_failure(p.status, gg::STATUS_TIMEOUT_EPILOGUE);
        }
        break;
      }
      ptx::tc_fence_after_sync();
      __syncwarp();
      uint32_t r[32];
      ptx::tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(part * 32) << 16) + acc * TILE_ROWS, r);
      ptx::tmem_ld_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh->tmem_empty[acc]);
      T* dst = static_cast<T*>(p.out) + static_cast<long>(c.row0) * p.n + col;
#pragma unroll
      for (int j = 0; j < TILE_ROWS; ++j) {
        if (j < c.valid && on) dst[static_cast<long>(j) * p.n] = Cvt<T>::from_f(gg::act_fwd<ACT>(__uint_as_float(r[j]) + bias));
      }
      __syncwarp();
    }
  }

  __syncwarp();
  if (*abort_flag != 0) {
    // give copies that were already issued time to land before the shared memory goes away
    const unsigned long long t0 = ptx::globaltimer();
    while (ptx::globaltimer() - t0 < 200000ull) __nanosleep(1000);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <typename T, int ACT>
cudaError_t launch_one(const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int grid, cudaStream_t stream) {
  static std::mutex mu;   // the shared-memory attribute is per device
  static uint64_t configured = 0;
  auto kernel = narrow_gemm_kernel<T, ACT>;
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
  return launch_chained(kernel, dim3(grid), dim3(NUM_THREADS), SMEM_BYTES, stream, tw, tx, p);
}

template <typename T>
cudaError_t launch_act(int act, const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int grid, cudaStream_t stream) {
  switch (act) {
    case kActRelu: return launch_one<T, kActRelu>(tw, tx, p, grid, stream);
    case kActGelu: return launch_one<T, kActGelu>(tw, tx, p, grid, stream);
    case kActGeluTanh: return launch_one<T, kActGeluTanh>(tw, tx, p, grid, stream);
    default: return launch_one<T, kActNone>(tw, tx, p, grid, stream);
  }
}

}  // namespace

cudaError_t launch(int dtype, int act, const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int grid,
                   cudaStream_t stream) {
  return dtype == kBF16 ? launch_act<__nv_bfloat16>(act, tw, tx, p, grid, stream)
                        : launch_act<__half>(act, tw, tx, p, grid, stream);
}

}  // namespace ng
}  // namespace fmoe
