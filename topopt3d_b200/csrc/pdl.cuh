// Programmatic dependent launch.  A kernel launched by launch_pdl may have its
// blocks resident before the kernel ahead of it in the stream has finished;
// it calls pdl_wait before its first access to global memory, which returns
// when that kernel is complete and its writes are visible, and after that
// pdl_launch_dependents, so that the kernel behind it can be set up while it
// drains.  Since every such kernel waits first, the order of all accesses stays
// that of the stream; what overlaps is the launch.  Both calls do nothing in
// a kernel launched without the attribute.  With the fine
// operator, the transfers and CG's updates launched this way a solve of 12x6x6
// takes 0.06 ms less (of 0.75), of 48x24x24 0.05 (of 1.13), of 91x47x53 mixed
// 0.27 (of 3.34), of 192x96x96 0.3 to 0.6%.  The persistent coarse cycle does
// not release the prolongation early: its blocks beside the cycle's cost
// 91x47x53 0.06 ms.
#pragma once

#include <cuda_runtime.h>

namespace tpo {

__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<A &&>(args)...);
}

}  // namespace tpo
