// pdl.cuh -- programmatic dependent launch for the chains of short kernels.
//
// A solve of a few thousand rows is several hundred launches of 3 to 30 us, each
// starting 1.5 to 2 us after the last ended.  Launched by gb_pdl, a kernel's CTAs may
// become resident while the kernel before drains; gb_pdl_entry, its first statement,
// waits until that kernel has completed and its writes are visible, and then lets the
// next kernel start in the same way (its CTAs find room once every CTA of this one is
// resident).  Order and visibility are those of the stream.
#pragma once
#include <cuda_runtime.h>

static __device__ __forceinline__ void gb_pdl_entry()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// (launch errors are left for cudaGetLastError, as by <<<>>>)
template <typename... P, typename... A>
static inline void gb_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
