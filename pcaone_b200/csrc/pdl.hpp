// Programmatic dependent launch: a kernel of the window-run / Omega-update chain is launched while
// the one before it still runs and waits, before it touches any memory, until that one is
// complete, so its launch and its CTAs' start are hidden. The chain's kernels run for 5 to 30 us
// on the windows of small and ordinary panels, where that start is a tenth of the time.
//
// Every kernel launched with launch_pdl calls pdl_begin() before its first global memory access:
// it lets the next kernel start (all CTAs of this one are running or done by the time that
// happens, so none of them can be kept from its SM) and waits for the previous kernel, which
// itself waited for its own predecessor: everything queued before is complete.
//
// Such a kernel may be resident while the kernels before it still write their results, so what
// they wrote is not read-only for its lifetime: results of the chain (products, operands, G, H,
// Omega, factors, maxima) are read with ordinary loads, never __ldg and never through a
// `const T* __restrict__` parameter, which the compiler may turn into loads of the non-coherent
// path or move above the wait. Codes, the dense matrix and the missing-entry lists are
// complete before the chain's first kernel starts and may be read either way.
#pragma once

#include <cuda_runtime.h>

#include "internal.hpp"

namespace pg {

__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A result of the chain that the calling kernel does not write itself: an ordinary load that stays
// where it is written, so that a batch of them is in flight before the first is used (plain
// C++ loads were sunk to their uses: epilogues of a winSVD, N = 5003, M = 80021, l = 52, a quarter
// of the entries missing: 63.5 ms against 59.6).
__device__ __forceinline__ float4 chain_load(const float4* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
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
