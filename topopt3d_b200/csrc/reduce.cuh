// Deterministic grid reductions with an FP64 result: the blocks of a sum
// write one partial each, and the last block to finish (a ticket counter)
// sums them in a fixed order.  Used by the vector kernels (kernels_vec.cu)
// and by the dot products in the epilogue of the fine-level operator
// (kernels_apply_staged.cu).
#pragma once

namespace tpo {

// sum over a block of up to 1024 threads, valid in thread 0; tid is the
// linear thread index
__device__ __forceinline__ double block_sum(double v, double *sh, int tid, int threads) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = tid & 31, w = tid >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  v = 0;
  if (tid < 32) {
    v = (tid < (threads >> 5)) ? sh[tid] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  return v;
}

// partial of block `block` of `blocks` -> last block -> *out (previous *out
// moved to *shift_to if set); the ticket ends at zero
__device__ __forceinline__ void finish_reduction(double v, int tid, int threads, int block,
                                                 int blocks, double *part,
                                                 unsigned int *ticket, double *out,
                                                 double *shift_to) {
  __shared__ double sh[32];
  __shared__ bool last;
  v = block_sum(v, sh, tid, threads);
  if (tid == 0) {
    part[block] = v;
    __threadfence();
    last = (atomicAdd(ticket, 1u) == (unsigned int)blocks - 1u);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s = 0;
  for (int i = tid; i < blocks; i += threads) s += ((volatile double *)part)[i];
  s = block_sum(s, sh, tid, threads);
  if (tid == 0) {
    if (shift_to) *shift_to = *out;
    *out = s;
    *ticket = 0u;
  }
}

}  // namespace tpo
