// Programmatic dependent launch.  A kernel launched by launch_pdl may have its
// blocks resident before the kernel ahead of it in the stream has finished.
// Its rules:
//
// * All of its blocks call pdl_wait before their first access to anything that
//   a kernel of the stream writes; the call returns when the kernel ahead is
//   complete and its writes are visible.  So a kernel's completion stands for all
//   before it, and the order of all accesses stays that of the stream; what
//   overlaps is the launch.  Before the wait a kernel may read what was there
//   before the whole chain: the inversion's kernels (kernels_coarse_inv.cu) read
//   their task lists, which are uploaded once per context.
// * A block calls pdl_launch_dependents after its last store to a vector that the
//   kernel behind reads by load_ro.  The blocks of that kernel start when every
//   block has made the call, so its operands are not written while it lives.  A
//   sum that the last block writes (finish_reduction) comes after the call, and
//   the inversion's kernels make theirs before their stores: such values are
//   read through plain pointers or cp.async.
// * __ldg and const __restrict__ operands are not used.  Their loads may be moved
//   above the wait; load_ro is the same read-only load, kept in its place.
//   (Read-only loads are worth having: with plain ones the fine operator's
//   L2 traffic is half as much again, and its product takes 65 us for 58 in
//   FP64, 33 for 30.5 in FP32 at 192x96x96.)
//
// Both calls do nothing in a kernel launched without the attribute.
//
// The level-1 pair (kernels_l1tc.cu) is the exception.  k_l1_corr_apply releases
// at its start, and k_apply_l1_tc behind it reads u and the moduli, and writes y
// in blocks without correction rows, before it waits.  That is sound because
// k_l1_corr_apply is launched WITHOUT the attribute: all before it is complete
// when it starts, and it writes nothing but the correction values, which the
// kernel behind reads after its wait, through plain pointers.
//
// With the fine operator, the transfers and CG's updates launched this way a
// solve of 12x6x6 takes 0.06 ms less (of 0.75), of 48x24x24 0.05 (of 1.13), of
// 91x47x53 mixed 0.27 (of 3.34), of 192x96x96 0.3 to 0.6%.  The persistent
// coarse cycle does not release the prolongation early: its blocks beside the
// cycle's cost 91x47x53 0.06 ms.
#pragma once

#include <cuda_runtime.h>

namespace tpo {

__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// *p through the read-only path, not before what comes ahead of it here
__device__ __forceinline__ float load_ro(const float *p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double load_ro(const double *p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned load_ro(const unsigned char *p) {
  unsigned v;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 load_ro(const float4 *p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ double2 load_ro(const double2 *p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
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
