// Programmatic dependent launch: a kernel of the window-run / Omega-update chain is launched while
// the one before it still runs and waits, before it touches any memory, until that one is
// complete, so its launch and its CTAs' start are hidden. The chain's kernels run for 5 to 30 us
// on the windows of small and ordinary panels, where that start is a tenth of the time.
//
// Every kernel launched with launch_pdl calls pdl_begin() before its first global memory access:
// it lets the next kernel start (all CTAs of this one are running or done by the time that
// happens, so none of them can be kept from its SM) and waits for the previous kernel, which
// itself waited for its own predecessor: everything queued before is complete.
#pragma once

#include <cuda_runtime.h>

#include "internal.hpp"

namespace pg {

__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... KArgs, typename... Args>
void launch_pdl(void (*kern)(KArgs...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  PG_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
}

}  // namespace pg
