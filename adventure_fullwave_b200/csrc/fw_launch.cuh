// Launch of one kernel of an iteration's chain.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace fw {

// Programmatic dependent launch: the kernel may be set up on the SMs that the
// one before it leaves free, and waits in chain_begin() for its results.  An
// iteration is six to ten short kernels, each needing the one before; started
// one after another their launch latency and first instructions are a third
// of a small model's iteration.  `kernel` must begin with chain_begin().
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                           A &&...args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);  // (checked by cudaGetLastError)
}

}  // namespace fw
