// f16 instantiations of the grouped GEMM for few or ragged rows.
#include "slim_gemm_kernel.cuh"

namespace fmoe {
namespace slim {
cudaError_t launch_f16(int mode, int act, const Maps& m, const Params& p, int grid, cudaStream_t stream) {
  return launch_for_type<__half>(mode, act, m, p, grid, stream);
}
}  // namespace slim
}  // namespace fmoe
