// Host side of the tcgen05 grouped GEMM: tensor-map construction and dispatch.  The kernels live
// in slim_gemm_kernel.cuh (CTA pairs, most row modes), pair_gemm_kernel.cuh (CTA pairs, weight
// gradients), grouped_gemm_kernel.cuh (row modes with rows arriving from or leaving for other GPUs) —
// instantiated per element type in slim_gemm_*.cu / pair_gemm_*.cu / grouped_gemm_*.cu — and
// narrow_gemm.cu (decoding).
#include <algorithm>

#include "grouped_gemm_kernel.cuh"
#include "narrow_gemm.cuh"
#include "pair_gemm_kernel.cuh"
#include "slim_gemm_kernel.cuh"
#include "tensor_map.cuh"

namespace fmoe {
using namespace gg;
namespace {

// ------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
  });
  return fn;
}

bool encode(CUtensorMap* map, int dtype, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
            const cuuint32_t* box) {
  const bool half_line = box[0] * 2 == 64;   // 32 columns: 64-byte swizzle
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return false;
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, dtype == kBF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                      : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                  rank, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, half_line ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

bool make_map_2d(CUtensorMap* map, int dtype, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                 uint32_t box_outer) {
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {inner * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  return encode(map, dtype, base, 2, dims, strides, box);
}

bool make_map_3d(CUtensorMap* map, int dtype, const void* base, uint64_t inner, uint64_t mid, uint64_t outer,
                 uint32_t box_inner, uint32_t box_mid) {
  cuuint64_t dims[3] = {inner, mid, outer};
  cuuint64_t strides[2] = {inner * 2, mid * inner * 2};
  cuuint32_t box[3] = {box_inner, box_mid, 1};
  return encode(map, dtype, base, 3, dims, strides, box);
}

bool make_map_columns(CUtensorMap* map, int dtype, const void* base, uint64_t inner, uint64_t outer, uint32_t box_outer,
                      uint32_t box_blocks) {
  cuuint64_t dims[3] = {64, outer, inner / 64};
  cuuint64_t strides[2] = {inner * 2, 128};
  cuuint32_t box[3] = {64, box_outer, box_blocks};
  return encode(map, dtype, base, 3, dims, strides, box);
}

bool grouped_gemm_supported(int mode, int m, int n, int k, int num_groups) {
  if (num_groups < 1 || num_groups > MAX_GROUPS) return false;
  if (n % 32 != 0 || n < 32) return false;
  if (mode == kWgrad) return m % 8 == 0 && m >= 8;
  return k % 64 == 0 && k >= 64;
}

namespace {

bool exchanges(const GroupedGemmArgs& a) {
  return a.send.enabled || a.gate.flags != nullptr || a.push_meta != nullptr || a.trace != nullptr;
}

// A handful of rows per expert and nothing saved for a backward: the weights' bytes are the work
// (64 experts, 128 rows, 1024 <-> 4096: 74 and 74 us against 85 and 82 of the single-CTA kernel; 8
// experts, 16 rows: 15 and 23 against 22 and 27).  Up to 256 rows in all: with 1024 rows that go to
// two of 64 experts every 32-row tile reads the weights again, 43 against 19 us.
bool narrow_applies(const GroupedGemmArgs& a) {
  return a.mode == kRowsNT && a.epi == kEpiBiasAct && a.pre_out == nullptr && a.rows_cap <= 256 &&
         a.rows_cap <= 16L * a.num_groups && !exchanges(a);
}

// The kernel with the token rows on the N side takes nearly all row modes without an exchange.  us, it
// against the kernel of 256-row tiles, forward with GELU and saved pre-activation / forward without /
// input gradient with the derivative / without: 1024 <-> 4096, 64 experts, 128 rows each: 122, 114, 117,
// 110 against 133, 124, 133, 120; 8 experts, 64 rows each: 17.5, 24.6, 18.3, 24.5 against 22.6, 26.1,
// 22.1, 25.7; 8 experts, 750 rows each: 54, 50, 56, 49 against 56, 53, 56, 52; 512 <-> 2048, 64 experts,
// 64 rows each: 36, 32, 36, 32 against 55, 35, 54, 34.  With up to 16 rows per expert against the
// single-CTA kernel: 512 <-> 2048, 8 experts: 7.7, -, 7.7, 13.7 against 15.6, -, 13.6, 16.0.
// The others stay where they are better: with few rows per expert, no activation and more tiles than
// pairs the single-CTA kernel shares the weights' bytes more evenly (64 experts, 4 rows each, 4096 ->
// 1024: 94 against 82), and with many rows the derivative's chunks need not be transposed (2 experts,
// 4096 rows each: 69.0 against 67.3; 4915 rows each: 81 against 78).
bool slim_applies(const GroupedGemmArgs& a) {
  if (a.mode == kWgrad || exchanges(a)) return false;
  const bool plain = a.act == kActNone;
  if (a.mode == kRowsNT ? a.epi != kEpiBiasAct
                        : a.bias != nullptr || a.pre_out != nullptr || !(plain || (a.epi == kEpiDAct && a.aux != nullptr))) {
    return false;
  }
  if (plain && a.rows_cap <= 16L * a.num_groups) {
    return static_cast<long>(a.num_groups) * ((a.n + slim::TILE_N - 1) / slim::TILE_N) <= a.num_sms / 2;
  }
  return a.mode == kRowsNT || plain || a.rows_cap <= 512L * a.num_groups;
}

// The paired kernel of 256-row tiles: weight gradients, and the derivative of many rows.
bool pair_applies(const GroupedGemmArgs& a) {
  if (a.mode == kWgrad) return true;
  return a.mode == kRowsNN && !exchanges(a) && a.rows_cap > 512L * a.num_groups && a.bias == nullptr &&
         a.pre_out == nullptr && a.act != kActNone && a.epi == kEpiDAct && a.aux != nullptr;
}

// Whether the column sums of a weight gradient end before its main loops when one warp per CTA forms them.  In
// us: an item of 32 columns takes 1.7 and 0.9 more per 128 rows, a tile 0.6 per 64 rows and not less than 2.1.  The
// epilogue warps' sums against that warp's (launch with the sums, us): 8 experts, 2048 rows, 2048 x 256: 21
// against 73, x 512: 36, 72, x 1024: 64, 61; 8 of 1000, 4096 x 256: 24, 68, x 512: 39, 69, x 1024: 63, 60; 16 of 512,
// 1024 x 256: 10, 16, x 1024: 21, 20; 16 of 64, 1024 x 1024: 13.0, 10.8; 2 of 4096, 4096 x 1024: 60, 57; 1 of 8192,
// 64 x 1024: 59, 50.  The margin of 1.3 is for rows that are in the L2.
bool sums_beside(const GroupedGemmArgs& a, int grid) {
  const long rows = (a.rows_cap + a.num_groups - 1) / a.num_groups;
  const long items = static_cast<long>(a.num_groups) * ((a.m + pg::SUM_COLS - 1) / pg::SUM_COLS);
  const long tiles = static_cast<long>(a.num_groups) * ((a.m + pg::TILE_M - 1) / pg::TILE_M) * ((a.n + pg::TILE_N - 1) / pg::TILE_N);
  const double item = 1.7 + 0.9 * static_cast<double>((rows + 127) / 128);
  const double tile = std::max(2.1, 0.6 * static_cast<double>((rows + BK - 1) / BK));
  return static_cast<double>((items + grid - 1) / grid) * item <= 1.3 * static_cast<double>((tiles + grid / 2 - 1) / (grid / 2)) * tile;
}

template <typename P> void set_offsets(P& p, const GroupedGemmArgs& a) {
  p.offs = a.offs;
  p.one_group[0] = 0;
  p.one_group[1] = static_cast<int>(a.rows_cap);
}

cudaError_t launch_narrow_gemm(const GroupedGemmArgs& a) {
  CUtensorMap tw, tx;
  if (!make_map_2d(&tw, a.dtype, a.b, a.k, static_cast<uint64_t>(a.num_groups) * a.n, ng::BK, ng::TILE_N) ||
      !make_map_2d(&tx, a.dtype, a.a, a.k, a.rows_cap, ng::BK, ng::TILE_ROWS)) {
    return cudaErrorInvalidValue;
  }
  ng::Params p;
  p.num_groups = a.num_groups;
  p.n = a.n;
  p.k = a.k;
  set_offsets(p, a);
  p.bias = a.bias;
  p.out = a.out;
  p.status = a.status;
  return ng::launch(a.dtype, a.act, tw, tx, p, a.num_sms > 0 ? a.num_sms : 148, a.stream);
}

cudaError_t launch_slim_gemm(const GroupedGemmArgs& a) {
  slim::Maps m;
  const uint64_t groups = a.num_groups;
  const bool blocks = a.mode == kRowsNN && a.n % 64 == 0;
  bool ok = make_map_3d(&m.c, a.dtype, a.out, a.n, a.rows_cap, 1, 32, 32);
  if (a.mode == kRowsNT) {
    ok = ok && make_map_2d(&m.w, a.dtype, a.b, a.k, groups * a.n, BK, slim::CTA_N);
  } else if (blocks) {
    ok = ok && make_map_columns(&m.w, a.dtype, a.b, a.n, groups * a.k, BK, 2);
  } else {
    ok = ok && make_map_2d(&m.w, a.dtype, a.b, a.n, groups * a.k, 64, BK);
  }
  for (int i = 0; i < slim::HALF_SIZES; ++i) {
    ok = ok && make_map_2d(&m.x[i], a.dtype, a.a, a.k, a.rows_cap, BK, (i + 1) * slim::HALF_STEP);
  }
  if (!ok) return cudaErrorInvalidValue;
  slim::Params p;
  p.num_groups = a.num_groups;
  p.n = a.n;
  p.k = a.k;
  p.w_blocks = blocks ? 1 : 0;
  set_offsets(p, a);
  p.out = a.out;
  p.pre_out = a.pre_out;
  p.bias = a.bias;
  p.aux = a.aux;
  p.status = a.status;
  const int grid = (a.num_sms > 1 ? a.num_sms : 148) & ~1;
  return a.dtype == kBF16 ? slim::launch_bf16(a.mode, a.act, m, p, grid, a.stream)
                          : slim::launch_f16(a.mode, a.act, m, p, grid, a.stream);
}

cudaError_t launch_pair_gemm(const GroupedGemmArgs& a) {
  CUtensorMap ta, tb, tc;
  // (an fp32 or accumulated gradient is not stored through the map)
  bool ok = a.mode == kWgrad ? make_map_3d(&tc, a.dtype, a.out, a.n, a.m, a.num_groups, 64, 32)
                             : make_map_3d(&tc, a.dtype, a.out, a.n, a.rows_cap, 1, 64, 32);
  if (!ok) return cudaErrorInvalidValue;
  if (a.mode == kRowsNN) {
    ok = make_map_2d(&ta, a.dtype, a.a, a.k, a.rows_cap, BK, pg::CTA_M) &&
         make_map_2d(&tb, a.dtype, a.b, a.n, static_cast<uint64_t>(a.num_groups) * a.k, 64, BK);
  } else {
    ok = make_map_2d(&ta, a.dtype, a.a, a.m, a.rows_cap, 64, BK) &&
         make_map_2d(&tb, a.dtype, a.b, a.n, a.rows_cap, 64, BK);
  }
  if (!ok) return cudaErrorInvalidValue;
  pg::Params p;
  p.num_groups = a.num_groups;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  set_offsets(p, a);
  p.out = a.out;
  p.aux = a.aux;
  p.accumulate = a.accumulate;
  p.out_fp32 = a.out_fp32;
  p.psum = a.mode == kWgrad ? a.psum : nullptr;
  p.psrc = a.a;
  p.qsrc = a.b;
  p.status = a.status;
  const int grid = (a.num_sms > 1 ? a.num_sms : 148) & ~1;
  p.side_sums = p.psum != nullptr && sums_beside(a, grid) ? 1 : 0;
  return a.dtype == kBF16 ? pg::launch_bf16(a.mode, a.act, ta, tb, tc, p, grid, a.stream)
                          : pg::launch_f16(a.mode, a.act, ta, tb, tc, p, grid, a.stream);
}

}  // namespace

cudaError_t launch_grouped_gemm(const GroupedGemmArgs& a) {
  if (!grouped_gemm_supported(a.mode, a.m, a.n, a.k, a.num_groups)) return cudaErrorInvalidValue;
  if (a.offs == nullptr && a.num_groups != 1) return cudaErrorInvalidValue;
  if (a.rows_cap == 0) {
    // no rows: no tensor map has an extent of 0.  The weight gradient is the empty sum.
    if (a.mode != kWgrad || a.accumulate) return cudaSuccess;
    const size_t width = static_cast<size_t>(a.num_groups) * a.m;
    const cudaError_t e = cudaMemsetAsync(a.out, 0, width * a.n * (a.out_fp32 ? 4 : 2), a.stream);
    if (e != cudaSuccess || a.psum == nullptr) return e;
    return cudaMemsetAsync(a.psum, 0, width * 2, a.stream);
  }
  if (narrow_applies(a)) return launch_narrow_gemm(a);
  if (slim_applies(a)) return launch_slim_gemm(a);
  if (pair_applies(a)) return launch_pair_gemm(a);
  CUtensorMap ta, tb;
  bool ok = true;
  if (a.mode == kRowsNT) {
    ok = make_map_2d(&ta, a.dtype, a.a, a.k, a.rows_cap, BK, BM) &&
         make_map_2d(&tb, a.dtype, a.b, a.k, static_cast<uint64_t>(a.num_groups) * a.n, BK, BN);
  } else {
    ok = make_map_2d(&ta, a.dtype, a.a, a.k, a.rows_cap, BK, BM) &&
         make_map_2d(&tb, a.dtype, a.b, a.n, static_cast<uint64_t>(a.num_groups) * a.k, 64, BK);
  }
  if (!ok) return cudaErrorInvalidValue;

  KernelParams kp;
  kp.num_groups = a.num_groups;
  kp.n = a.n;
  kp.k = a.k;
  set_offsets(kp, a);
  kp.out = a.out;
  kp.pre_out = a.pre_out;
  kp.bias = a.bias;
  kp.aux = a.aux;
  kp.act = a.act;
  kp.epi = a.epi;
  kp.status = a.status;
  kp.push_meta = a.push_meta;
  kp.push_dst = a.push_dst;
  kp.push_flags = a.push_flags;
  kp.push_epoch = a.push_epoch;
  kp.push_counter = a.push_counter;
  kp.push_me = a.push_me;
  kp.push_world = a.push_world;
  kp.push_slots = a.push_slots;
  kp.send = a.send;
  kp.gate = a.gate;
  kp.trace = a.trace;
  if (kp.send.enabled && (kp.send.d % 8 != 0 || kp.send.item_prefix == nullptr ||
                          kp.send.item_count == nullptr)) {
    return cudaErrorInvalidValue;
  }

  const int grid = a.num_sms > 0 ? a.num_sms : 148;
  return a.dtype == kBF16 ? gg::launch_bf16(a.mode, ta, tb, kp, grid, a.stream)
                          : gg::launch_f16(a.mode, ta, tb, kp, grid, a.stream);
}

}  // namespace fmoe
