// Programmatic dependent launch: a kernel whose CTAs may start before the previous
// kernel of the stream has ended, does what does not depend on it, and waits.
#pragma once

#include <cuda_runtime.h>

namespace fd {

// The kernels before this one in the stream have ended, and their writes are
// visible (to loads that do not hit older lines of the SM's L1: ld.global.cg, TMA).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel of the stream may start.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch a kernel; `early`: its CTAs may start before the previous kernel of the
// stream has ended (the kernel must call pdl_wait).
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kern)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st, bool early,
                       A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace fd
