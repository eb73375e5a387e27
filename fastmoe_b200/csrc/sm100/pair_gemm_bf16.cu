// bf16 instantiations of the paired grouped GEMM kernel.
#include "pair_gemm_kernel.cuh"

namespace fmoe {
namespace pg {
cudaError_t launch_bf16(int mode, int act, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p, int grid,
                        cudaStream_t stream) {
  return launch_for_type<__nv_bfloat16>(mode, act, ta, tb, tc, p, grid, stream);
}
}  // namespace pg
}  // namespace fmoe
