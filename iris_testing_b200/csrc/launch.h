// Host side of programmatic dependent launch (see chain_wait in sm100_ptx.cuh).
#pragma once
#include <cuda_runtime.h>
#include <string.h>

namespace b200 {

inline cudaLaunchAttribute chained_attribute() {
  cudaLaunchAttribute a;
  memset(&a, 0, sizeof(a));
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

// Launches a kernel whose every thread calls chain_wait() before it touches what earlier kernels left.
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  A... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = chained_attribute();
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace b200
