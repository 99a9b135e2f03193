// markers.cuh -- the byte a window marker names (resolve.cu; plain C++ too, so
// that chains of any length can be checked on the CPU).
#pragma once
#include <cstdint>

#include "common.cuh"

#ifdef __CUDACC__
#define GZGPU_HD __host__ __device__ __forceinline__
#else
#define GZGPU_HD inline
#endif

namespace gzgpu {

// What a marker walk needs of a chunk: where its output begins, and its last
// two pages, which hold the 32 KiB that the chunk after it can name.
struct NearChunk {
  uint64_t out_off;
  uint32_t last_seq, last_page, prev_page, pad;
};
constexpr uint32_t kNear = 8;  // chunks before a unit's kept at hand

GZGPU_HD NearChunk near_chunk(const PlacedChunk& c) {
  return NearChunk{c.out_off, c.last_seq, c.last_page, c.prev_page, 0};
}

// The byte that marker v of placed chunk k, at output offset `off`, names:
// the one 65536 - v before the chunk, or 0 before the member's first byte
// (`moff`).  An entry found there that is a marker of its own chunk goes on
// from that chunk's start, so a chain can lead back over the whole member:
// offsets are 64-bit throughout.  near: the kNear chunks before k, nearest
// first; entry(page, i): entry i of a page.
template <typename Entry>
GZGPU_HD uint32_t follow_marker(const PlacedChunk* placed, const NearChunk* near, uint32_t k,
                                uint64_t off, uint64_t moff, uint32_t v, Entry entry) {
  uint32_t back = 0;  // chunks gone back from k
  for (;;) {
    const uint32_t dist = 2 * kMarkerBase - v;
    if (dist > off - moff) return 0;
    const uint64_t src = off - dist;
    NearChunk c;
    do {
      c = back < kNear ? near[back] : near_chunk(placed[k - 1 - back]);
      back++;
    } while (c.out_off > src);
    const uint64_t q = src - c.out_off;  // one of its last 32 Ki entries
    v = entry((uint32_t)(q >> 16) == c.last_seq ? c.last_page : c.prev_page, (uint32_t)q & (kPageEntries - 1));
    if (v < kMarkerBase) return v;
    off = c.out_off;
  }
}

}  // namespace gzgpu
