// Programmatic dependent launch for the hot kernels.
//
// A kernel launched this way may have its CTAs placed on SMs while the
// previous kernel in the stream drains, so launch latency and the kernel's
// own set-up overlap that kernel's last CTAs.  Every kernel launched through
// launch_pdl calls griddep_wait() (ptx.cuh) before its first access to memory
// that a kernel may write (tables of the plan, which none writes, may be read
// earlier), which holds it until the previous kernel has completed and its
// writes are visible: stream order is unchanged for the data.
// PLFFT_B200_NO_PDL=1 launches without the attribute.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <utility>

namespace plfft_b200 {

inline bool pdl_enabled() {
  static const bool on = std::getenv("PLFFT_B200_NO_PDL") == nullptr;
  return on;
}

// carveout: percent of an SM's memory to be shared memory, 0 for the driver's
// choice by the kernel's occupancy
template <class... Params, class... Args>
cudaError_t launch_pdl_carved(int carveout, void (*kern)(Params...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  if (carveout) {
    attr[cfg.numAttrs].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[cfg.numAttrs++].val.sharedMemCarveout = unsigned(carveout);
  }
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

template <class... Params, class... Args>
cudaError_t launch_pdl(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       Args&&... args) {
  return launch_pdl_carved(0, kern, grid, block, smem, st, std::forward<Args>(args)...);
}

}  // namespace plfft_b200
