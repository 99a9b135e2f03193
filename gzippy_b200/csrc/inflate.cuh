// inflate.cuh -- launch interface of the chunk inflate kernels.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace gzgpu {

constexpr int kRingWarps = 1;      // ring kernel: warps per CTA (64 KB ring each)
constexpr int kCtaThreads = 256;    // page kernel: threads per CTA (one chunk each)
constexpr int kWideThreads = 1024;  // the same in jobs of few chunks (one CTA per SM)
constexpr int kDistBits = 8;       // distance LUT index bits (ring kernel, sync-start search)

// page kernel: `ctas` (3 or 4) CTAs per SM; registers are sized for that many
// (80 or 64 per thread).  Also sets the kernels up for launch_inflate.
template <int LB>
int inflate_blocks_per_sm(bool ring, int ctas);
// wide: CTAs of kWideThreads; *n_sync (device): sync starts in the job (then
// successors are watched mid-block)
template <int LB>
cudaError_t launch_inflate(bool ring, int ctas, bool wide, const uint8_t* in, ChunkDesc* descs,
                           ChunkResult* results, const uint32_t* work, const uint32_t* n_work,
                           uint32_t* work_counter, const uint32_t* n_sync, const PagePool& pool,
                           int blocks, cudaStream_t stream);
// sync starts inside dynamic blocks for the listed pieces left without a start
cudaError_t launch_dyn_sync(const uint8_t* in, ChunkDesc* descs, const uint32_t* pieces, uint32_t n,
                            uint32_t* n_sync, cudaStream_t stream);

}  // namespace gzgpu
