// Launch of a kernel that begins with ptx::chain_begin(): programmatic stream serialisation, so that
// its blocks take the SMs the kernel before it leaves and its set-up overlaps that kernel's end.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace fmoe {

template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  if (e != cudaSuccess) cudaGetLastError();   // reported here, not by whoever asks next
  return e;
}

}  // namespace fmoe
