// barrier.cuh -- barriers of a CTA.
#pragma once

namespace gzgpu {

// All lanes of a warp have to reach a barrier of the CTA together.  After a
// loop whose lanes leave it at different times, or a branch that some of them
// take, they need not be: a warp barrier joins them first.  So every barrier
// of the CTA is one of these.
__device__ __forceinline__ void cta_sync() {
  __syncwarp();
  __syncthreads();
}
__device__ __forceinline__ bool cta_sync_or(bool p) {
  __syncwarp();
  return __syncthreads_or(p) != 0;
}
__device__ __forceinline__ int cta_sync_count(bool p) {
  __syncwarp();
  return __syncthreads_count(p);
}

}  // namespace gzgpu
