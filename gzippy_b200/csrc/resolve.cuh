// resolve.cuh -- launch interface of marker resolution and CRC.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace gzgpu {

cudaError_t resolve_init(cudaStream_t stream);
// every placed chunk's bytes, markers resolved, from the pages [0, n_pages).
// tails (for kTwoPass bytes of output and more): the placed chunks whose entries
// from body_end on are resolved before the others
constexpr uint64_t kTwoPass = 16u << 20;
constexpr uint32_t kTailUnit = 512;                       // body_end is a multiple of it, or all
constexpr uint32_t kTailUnits = kWindow / kTailUnit + 1;  // a tail's, at most
cudaError_t launch_resolve(const PlacedChunk* placed, const uint32_t* placed_of_chunk,
                           const uint32_t* tails, uint32_t n_tails, uint32_t n_pages,
                           const ChunkResult* results, const PagePool& pool, uint8_t* out,
                           cudaStream_t stream);
// CRC: one CTA per block of up to kCrcBlock bytes, a slice of kCrcSlice per thread
constexpr int kCrcThreads = 512;
constexpr uint32_t kCrcSlice = 128;
constexpr uint32_t kCrcBlock = kCrcSlice * kCrcThreads;
constexpr int kCrcCtasPerSm = 2;
constexpr int kCrcLevels = 9;  // log2(512 slices)
constexpr uint32_t kCrcTurns = 64;  // blocks of a CTA whose warps' registers are kept
// shared memory: 32 lane copies of the byte table, shift tables, the warps' registers
constexpr size_t kCrcSmem =
    256 * 32 * 4 + kCrcLevels * 4 * 256 * 4 + kCrcTurns * (kCrcThreads / 32) * 4;

// mem_end[m]: output offset just past member m; mem_raw[m]: its CRC register
// accumulator (zeroed before the launch); then each member's status
cudaError_t launch_crc(const CrcBlock* blocks, uint32_t n_blocks, const uint8_t* out,
                       const uint64_t* mem_end, uint32_t* mem_raw, const uint64_t* mem_trailer,
                       const uint64_t* mem_len, uint32_t n_mem, const uint8_t* in,
                       int32_t* mem_status, int sms, cudaStream_t stream);

}  // namespace gzgpu
