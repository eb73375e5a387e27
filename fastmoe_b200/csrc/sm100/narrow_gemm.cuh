// Interface of the grouped GEMM for a handful of rows per expert (narrow_gemm.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace fmoe {
namespace ng {

constexpr int TILE_N = 128;     // output columns (rows of W) per tile
constexpr int TILE_ROWS = 32;   // token rows per tile
constexpr int BK = 64;

struct Params {
  int num_groups;
  int n;
  int k;
  const int* offs;      // null: `one_group` instead
  int one_group[2];
  const void* bias;   // optional [num_groups, n]
  void* out;
  int* status;
};

// tw: W as [num_groups * n, k], box BK x TILE_N; tx: x as [rows, k], box BK x TILE_ROWS.
cudaError_t launch(int dtype, int act, const CUtensorMap& tw, const CUtensorMap& tx, const Params& p, int grid,
                   cudaStream_t stream);

}  // namespace ng
}  // namespace fmoe
