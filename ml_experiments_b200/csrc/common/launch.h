// Launch with programmatic stream serialisation: the kernel may start while the one before it in the stream ends, so that its launch and
// set-up (barriers, tensor memory, descriptors: 2 to 4 us) are hidden. It must call `after_previous` (ptx.cuh) in every block before it
// touches global memory or ends. For the kernels that a GPT block issues one after another; products back to back, 10007 x 768 x 768:
// 16.9 -> 14.5 us each, 49152 x 768 x 768: 53.3 -> 49.0 us; a 12-layer forward pass of 10007 tokens, 96 launches: 3.51 -> 3.40 ms.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace b200 {

template <typename... P, typename... A>
inline void launch_early(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);   // (the caller asks for the last error)
}

}  // namespace b200
