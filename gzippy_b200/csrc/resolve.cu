// resolve.cu -- window propagation, marker resolution and CRC32 (K3-K5).
//
// After decoding, every accepted chunk k has an output offset out_off[k]
// and u16 entries in its pages.  An entry v < 256 is a byte; v >= 32768 is
// window index v - 32768 of the 32 KiB that precede the chunk in the final
// output (replace_markers.rs:7-23), i.e. final[out_off - 32768 + v - 32768],
// read as 0 before the member's first byte (the zero window).
//
//   resolve      : every entry's byte.  A marker names a byte of the 32 KiB
//                  before its chunk, which lies in the tail (the last 32 KiB) of
//                  one of the few chunks before it; that entry is a literal or
//                  again a marker, naming a byte before its own chunk.  Each
//                  marker follows its references through the chunks' tails until
//                  it reaches a literal (or a position before the member: 0), so
//                  all chunks resolve in parallel and the window chain
//                  (window_map.rs:80-103, chunk_fetcher.rs
//                  publish_subchunk_windows :2295,
//                  resolve_and_narrow_markers_in_place_crc, chunk_data.rs:1745)
//                  needs no order
//   crc_blocks   : CRC32 of blocks of final output (up to 64 KiB of one
//                  member each), each block's CRC moved to its member's end
//                  and XORed into the member's register (crc32.rs
//                  combine_crc32 :127 combines the same quantities)
//   member_check : each member's CRC32 and ISIZE against its trailer
#include <cstdint>

#include "barrier.cuh"
#include "common.cuh"
#include "markers.cuh"
#include "resolve.cuh"

namespace gzgpu {

// One warp per unit of kResolveUnit entries of a page: literal bytes go to
// shared memory, markers to a list, which the lanes then follow one marker each
// (two dependent loads a reference), and the unit's bytes leave in aligned
// 16-byte stores.  The pass is instructions (94 per 32 entries of text, of which
// 40 % are markers of 1.4 references each) and scattered loads in between, so
// what counts is warps that never wait for each other: with units of 4096
// entries for a CTA of 256 threads, its three barriers cost a third of the time
// (64 MiB of text: 0.35 ms, 0.23 by warps).
//
// Where data repeats for longer than a chunk, every entry is a marker and its
// chain leads back over all chunks; following each to its end took 55 ms of 1 GiB
// of zeros in 43 chunks.  All that chains pass through are the chunks' tails, so
// a walk of more than one reference writes its byte over the marker it began at,
// if that lies in its chunk's tail, and later walks end there.
// Above kTwoPass bytes the tails (`tails`: their chunks' places) are a launch of
// their own, in output order, so that chunks in flight together take about the
// root of their number in references; a marker before them is then one load of
// the final output.  1 GiB of zeros 2.0 ms, 64 MiB of text 0.202 -> 0.175.  A
// second launch costs a smaller job more than that (12 MiB of noisy ramps: 21 us
// in one, 29 in two).  It may start while the first one's last CTAs run: it reads
// its entries and makes its lists, then waits for the tails (5 us less than one
// after the other).
enum ResolvePart { kResolveAll, kResolveTails, kResolveBodies };
constexpr uint32_t kResolveUnit = 512;
constexpr int kResolveThreads = 256;
constexpr uint32_t kResolveWarps = kResolveThreads / 32;
static_assert(kResolveUnit == 16 * 32, "16 entries a lane");
static_assert(kResolveUnit == kTailUnit, "the body ends at a unit's edge");

struct ResolveWarp {
  alignas(16) uint8_t bytes[kResolveUnit + 16];
  uint32_t list[kResolveUnit];  // entry << 16 | marker
  NearChunk near[kNear];        // the chunks before the unit's, nearest first
};

template <ResolvePart kPart>
__global__ void __launch_bounds__(kResolveThreads, 6)
    resolve_kernel(const PlacedChunk* __restrict__ placed, const uint32_t* __restrict__ placed_of_chunk,
                   const uint32_t* __restrict__ tails, uint32_t n_tails, uint32_t n_pages,
                   const ChunkResult* __restrict__ results, PagePool pool, uint8_t* out) {
  __shared__ ResolveWarp rw[kResolveWarps];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ResolveWarp& W = rw[warp];
  uint32_t k, page, first;  // the chunk, the page and the unit's first entry in it
  uint64_t q0, len;         // the same in the chunk, and where to stop
  if (kPart == kResolveTails) {
    cudaTriggerProgrammaticLaunchCompletion();
    const uint32_t id = blockIdx.x * kResolveWarps + warp;
    if (id >= n_tails * kTailUnits) return;
    k = tails[id / kTailUnits];
    const PlacedChunk& pc = placed[k];
    len = results[pc.chunk].out_len;
    q0 = pc.body_end + (id % kTailUnits) * kResolveUnit;
    page = (uint32_t)(q0 >> 16) == pc.last_seq ? pc.last_page : pc.prev_page;
    first = (uint32_t)q0 & (kPageEntries - 1);
  } else {
    // kResolveWarps units in a row; the first ones of every page, then the
    // next, ...: markers thin out along a chunk
    page = blockIdx.x % n_pages;
    first = ((blockIdx.x / n_pages) * kResolveWarps + warp) * kResolveUnit;
    const uint32_t cid = pool.owner[page], sw = pool.seq[page];
    k = placed_of_chunk[cid];
    q0 = (uint64_t)(sw & kSeqMask) * kPageEntries + first;
    // nothing of a chunk not accepted, or of a failed attempt's page
    len = 0;
    if (k != 0xFFFFFFFFu && (sw >> kGenShift) == results[cid].gen)
      len = kPart == kResolveAll ? results[cid].out_len : placed[k].body_end;
  }
  if (q0 >= len) {
    if (kPart == kResolveBodies) cudaGridDependencySynchronize();
    return;
  }
  const uint32_t n = (uint32_t)min((uint64_t)kResolveUnit, len - q0);
  uint16_t* const src = pool.data + (size_t)page * kPageEntries + first;
  uint4 x[2];
#pragma unroll
  for (uint32_t s = 0; s < 2; s++) {
    const uint32_t e = 8 * (lane + 32 * s);
    x[s] = e < n ? *reinterpret_cast<const uint4*>(src + e) : make_uint4(0, 0, 0, 0);
  }
  const uint64_t off = placed[k].out_off, moff = placed[k].member_off;
  if (kPart != kResolveBodies && lane < kNear && lane < k) W.near[lane] = near_chunk(placed[k - 1 - lane]);
  uint32_t n_list = 0;
#pragma unroll
  for (uint32_t s = 0; s < 2; s++) {
    const uint32_t e = 8 * (lane + 32 * s);
    *reinterpret_cast<uint2*>(W.bytes + e) =
        make_uint2(__byte_perm(x[s].x, x[s].y, 0x6420), __byte_perm(x[s].z, x[s].w, 0x6420));
    const uint32_t h[4] = {x[s].x, x[s].y, x[s].z, x[s].w};
    uint32_t m = 0;  // markers among the eight
#pragma unroll
    for (int i = 0; i < 4; i++) m |= ((h[i] >> 15 & 1) | (h[i] >> 30 & 2)) << (2 * i);
    if (e + 8 > n) m &= e < n ? (1u << (n - e)) - 1 : 0u;
    if (!__any_sync(0xFFFFFFFFu, m != 0)) continue;
    uint32_t at = __popc(m);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, at, d);
      if (lane >= d) at += v;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, at, 31);
    at += n_list - __popc(m);
    n_list += total;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if ((m >> i) & 1) W.list[at++] = (e + i) << 16 | ((h[i >> 1] >> (16 * (i & 1))) & 0xFFFFu);
  }
  __syncwarp();
  if (kPart == kResolveBodies) cudaGridDependencySynchronize();  // the tails are in place
  for (uint32_t i = lane; i < n_list; i += 32) {
    const uint32_t item = W.list[i];
    const uint32_t v = item & 0xFFFFu;
    uint32_t byte;
    if constexpr (kPart == kResolveBodies) {
      const uint32_t dist = 2 * kMarkerBase - v;
      byte = dist <= off - moff ? out[off - dist] : 0u;
    } else {
      uint32_t refs = 0;
      byte = follow_marker(placed, W.near, k, off, moff, v, [&](uint32_t p, uint32_t e) -> uint32_t {
        refs++;
        return __ldcg(pool.data + (size_t)p * kPageEntries + e);
      });
      if (refs > 1 && (kPart == kResolveTails || q0 + (item >> 16) + kWindow >= len)) src[item >> 16] = (uint16_t)byte;
    }
    W.bytes[item >> 16] = (uint8_t)byte;
  }
  __syncwarp();
  // the unit's bytes: aligned 16 of the output, then what lies around them
  uint8_t* const dst = out + off + q0;
  const uint32_t head = min((0u - (uint32_t)(off + q0)) & 15u, n);
  const uint32_t o = head + 16 * lane;  // this lane's first byte in the unit
  if (o + 16 <= n) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(W.bytes + (o & ~3u));
    const uint32_t sh = 8 * (o & 3);
    *reinterpret_cast<uint4*>(dst + o) =
        make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh),
                   __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
  }
  const uint32_t rest = head + ((n - head) & ~15u) + (lane & 15);
  if (lane < head) dst[lane] = W.bytes[lane];
  if (lane >= 16 && rest < n) dst[rest] = W.bytes[rest];
}

// ---------------------------------------------------------------------------
// CRC32 (reflected 0xEDB88320).  A CRC register s followed by n zero bytes
// becomes A^n(s) = s * x^(8n) mod P (linear in s), so
//   raw(M1 | M2) = A^|M2|(raw(M1)) ^ raw(M2)       (raw: register starts at 0)
//   crc(M)       = ~(A^|M|(0xFFFFFFFF) ^ raw(M))
// and leading zero bytes leave raw() unchanged (crc32.rs combine_crc32 :127
// combines the same quantities).  Each block's raw CRC is moved to its
// member's end with A^(bytes after the block) and XORed into the member's
// register, so blocks fold in independently, in any order.
// ---------------------------------------------------------------------------
__device__ uint32_t d_crc_tab[256];
__device__ uint32_t d_x2n[64];          // x^(2^k) mod P
// d_crc_shift[j][k][v] = A^(kCrcSlice << j)(v << 8k): moves a register past
// 2^j lane slices of zero bytes with 4 lookups
__device__ uint32_t d_crc_shift[kCrcLevels][4][256];

__device__ __forceinline__ uint32_t gf2_mulmod(uint32_t a, uint32_t b) {
  uint32_t r = 0;
#pragma unroll 8
  for (int i = 31; i >= 0; i--) {
    r ^= b & (0u - ((a >> i) & 1u));
    b = (b >> 1) ^ (0xEDB88320u & (0u - (b & 1u)));
  }
  return r;
}

// x^(8n) mod P
__device__ __forceinline__ uint32_t x_pow_8n(uint64_t n) {
  uint32_t p = 1u << 31;
  uint64_t e = n << 3;
  for (int k = 0; e; e >>= 1, k++)
    if (e & 1) p = gf2_mulmod(d_x2n[k & 63], p);
  return p;
}

// x^(8n) mod P computed by a whole warp: lane k takes exponent bits k and
// k + 32, then a product tree over the lanes (every lane gets the result)
__device__ __forceinline__ uint32_t x_pow_8n_warp(uint64_t n, int lane) {
  const uint64_t e = n << 3;
  uint32_t f = 1u << 31;
  if ((e >> lane) & 1) f = d_x2n[lane];
  if ((e >> (lane + 32)) & 1) f = gf2_mulmod(f, d_x2n[lane + 32]);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) f = gf2_mulmod(f, __shfl_xor_sync(0xFFFFFFFFu, f, d));
  return f;
}

__global__ void crc_init_kernel() {
  uint32_t i = threadIdx.x;
  uint32_t c = i;
  for (int k = 0; k < 8; k++) c = (c >> 1) ^ (0xEDB88320u & (0u - (c & 1u)));
  d_crc_tab[i] = c;
  if (i == 0) {
    uint32_t v = 1u << 30;  // x^1
    for (int k = 0; k < 64; k++) {
      d_x2n[k] = v;
      v = gf2_mulmod(v, v);
    }
  }
}

// one block per (level, byte slot): 256 register values each
__global__ void crc_shift_init_kernel() {
  const uint32_t j = blockIdx.x >> 2, k = blockIdx.x & 3, v = threadIdx.x;
  const uint32_t xp = x_pow_8n((uint64_t)kCrcSlice << j);
  d_crc_shift[j][k][v] = gf2_mulmod(xp, v << (8 * k));
}

// the register s moved past 2^j lane slices, from the shift tables in shared memory
__device__ __forceinline__ uint32_t crc_shift(const uint32_t* shf, uint32_t s, int j) {
  const uint32_t* t = shf + j * 1024;
  return t[s & 0xFF] ^ t[256 + ((s >> 8) & 0xFF)] ^ t[512 + ((s >> 16) & 0xFF)] ^ t[768 + (s >> 24)];
}

// the register moved past one byte (added to its low end before), from the
// lane's own copy of the byte table (word 32 * index + lane of the shared
// array: every lane of a warp reads its own bank)
__device__ __forceinline__ uint32_t crc_step(const uint32_t* ltab, uint32_t lane, uint32_t c) {
  return ltab[((c & 0xFFu) << 5) | lane] ^ (c >> 8);
}

// CRC32 of the final output, one CTA per block of up to kCrcBlock bytes of one
// member.  Blocks end on 16-byte boundaries of the output; the bytes before
// the member's first and after its last count as zeros (the first leave the
// register at 0, the others are taken back by member_check).  Every thread
// folds a slice of kCrcSlice bytes byte by byte with its lane's copy of the
// byte table (no bank conflicts), from aligned 16-byte loads; the slices'
// registers merge in a tree of fixed shifts, and the block's register, moved
// past the rest of its member, is XORed into mem_raw.  What a block waits for
// is the serial chain of its bytes (a table read each), so slices are short
// (with 1 KiB slices, a warp per 32 KiB, a 4 KiB stream took 50 us, now 9).
// The warps merge their own slices and leave their registers; the blocks are
// put together at the end, a warp each, so that no warp waits for another in
// between (the move past a member's rest alone is 6,000 cycles of one warp:
// 128 MiB took 113 us with it between the blocks, now 86).
__global__ void __launch_bounds__(kCrcThreads)
    crc_blocks_kernel(const CrcBlock* __restrict__ blocks, uint32_t n,
                      const uint8_t* __restrict__ out, uint32_t* __restrict__ mem_raw) {
  extern __shared__ __align__(16) uint32_t sm[];
  uint32_t* ltab = sm;                                // [256][32] lane copies of the byte table
  uint32_t* shf = sm + 256 * 32;                      // [kCrcLevels][4][256] shift tables
  uint32_t* part = shf + kCrcLevels * 4 * 256;        // [kCrcTurns][warps]
  constexpr int kWarps = kCrcThreads / 32;
  for (uint32_t i = threadIdx.x; i < 256 * 32; i += kCrcThreads) ltab[i] = d_crc_tab[i >> 5];
  for (uint32_t i = threadIdx.x; i < kCrcLevels * 256; i += kCrcThreads)
    reinterpret_cast<uint4*>(shf)[i] = reinterpret_cast<const uint4*>(&d_crc_shift[0][0][0])[i];
  cta_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t b0 = blockIdx.x; b0 < n; b0 += kCrcTurns * gridDim.x) {
    uint32_t turns = 0;
    for (uint32_t bi = b0; bi < n && turns < kCrcTurns; bi += gridDim.x, turns++) {
      const CrcBlock blk = blocks[bi];
      // this thread's slice [s0, s0 + kCrcSlice) of the output
      const int64_t s0 = (int64_t)blk.end - (int64_t)kCrcSlice * (kCrcThreads - (int)threadIdx.x);
      uint32_t c = 0;
      if (s0 + (int64_t)kCrcSlice > (int64_t)blk.begin) {
        uint4 v[kCrcSlice / 16];
#pragma unroll
        for (uint32_t i = 0; i < kCrcSlice / 16; i++) {
          const int64_t a = s0 + 16 * (int64_t)i;
          v[i] = a + 16 > (int64_t)blk.begin && a + 16 <= (int64_t)blk.last
                     ? *reinterpret_cast<const uint4*>(out + a)
                     : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (uint32_t i = 0; i < kCrcSlice / 16; i++) {
          uint32_t wd[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
          const int64_t a = s0 + 16 * (int64_t)i;
          if (a < (int64_t)blk.begin || a + 16 > (int64_t)blk.last) {
            // the ends: bytes outside the member count as zeros
#pragma unroll
            for (int k = 0; k < 16; k++) {
              const bool in = a + k >= (int64_t)blk.begin && a + k < (int64_t)blk.last;
              const uint32_t byte = in ? out[a + k] : 0u;
              wd[k >> 2] = (wd[k >> 2] & ~(0xFFu << (8 * (k & 3)))) | byte << (8 * (k & 3));
            }
          }
#pragma unroll
          for (int k = 0; k < 4; k++) {
            c ^= wd[k];
#pragma unroll
            for (int b = 0; b < 4; b++) c = crc_step(ltab, lane, c);
          }
        }
      }
      __syncwarp();
      // slices merge: 2^j slices on each side at level j, first in the warps
#pragma unroll
      for (int j = 0; j < 5; j++) {
        const uint32_t r = __shfl_down_sync(0xFFFFFFFFu, c, 1 << j);
        if ((lane & ((2 << j) - 1)) == 0) c = crc_shift(shf, c, j) ^ r;
      }
      if (lane == 0) part[turns * kWarps + warp] = c;
    }
    cta_sync();
    for (uint32_t t = warp; t < turns; t += kWarps) {
      const CrcBlock blk = blocks[b0 + t * gridDim.x];
      uint32_t c = lane < kWarps ? part[t * kWarps + lane] : 0u;
#pragma unroll
      for (int j = 0; (1 << j) < kWarps; j++) {
        const uint32_t r = __shfl_down_sync(0xFFFFFFFFu, c, 1 << j);
        if ((lane & ((2 << j) - 1)) == 0) c = crc_shift(shf, c, 5 + j) ^ r;
      }
      if (blk.after) c = gf2_mulmod(x_pow_8n_warp(blk.after, lane), c);
      if (lane == 0) atomicXor(mem_raw + blk.member, c);
    }
    cta_sync();
  }
}

// one warp per member: its CRC from the accumulated blocks, checked with the
// trailer's CRC32 and ISIZE.  mem_end: the output offset past its last byte.
__global__ void member_check_kernel(const uint64_t* __restrict__ mem_trailer,
                                    const uint64_t* __restrict__ mem_len,
                                    const uint64_t* __restrict__ mem_end, uint32_t n_mem,
                                    const uint8_t* __restrict__ in,
                                    const uint32_t* __restrict__ mem_raw, int32_t* __restrict__ mem_status) {
  const uint32_t m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= n_mem) return;
  const uint64_t t = mem_trailer[m], len = mem_len[m];
  int32_t st = kOk;
  if (t != kNoTrailer) {
    // the register ran over `pad` zero bytes past the member; x^(2^32 - 1) = 1
    // mod P, so x^(8 (2^32 - 1 - pad)) takes them back
    const uint32_t pad = (uint32_t)(0 - mem_end[m]) & 15;
    uint32_t raw = mem_raw[m];
    if (pad) raw = gf2_mulmod(x_pow_8n_warp(0xFFFFFFFFull - pad, lane), raw);
    const uint32_t crc = ~(gf2_mulmod(x_pow_8n_warp(len, lane), 0xFFFFFFFFu) ^ raw);
    const uint32_t ecrc = in[t] | (in[t + 1] << 8) | ((uint32_t)in[t + 2] << 16) | ((uint32_t)in[t + 3] << 24);
    const uint32_t eisz = in[t + 4] | (in[t + 5] << 8) | ((uint32_t)in[t + 6] << 16) | ((uint32_t)in[t + 7] << 24);
    if ((uint32_t)len != eisz) st = kSizeMismatch;
    else if (crc != ecrc) st = kCrcMismatch;
  }
  if (lane == 0) mem_status[m] = st;
}

cudaError_t resolve_init(cudaStream_t stream) {
  crc_init_kernel<<<1, 256, 0, stream>>>();
  crc_shift_init_kernel<<<4 * kCrcLevels, 256, 0, stream>>>();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(crc_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kCrcSmem);
}

cudaError_t launch_resolve(const PlacedChunk* placed, const uint32_t* placed_of_chunk,
                           const uint32_t* tails, uint32_t n_tails, uint32_t n_pages,
                           const ChunkResult* results, const PagePool& pool, uint8_t* out,
                           cudaStream_t stream) {
  const uint32_t body_ctas = n_pages * (kPageEntries / (kResolveUnit * kResolveWarps));
  if (!body_ctas) return cudaSuccess;
  if (!n_tails) {
    resolve_kernel<kResolveAll><<<body_ctas, kResolveThreads, 0, stream>>>(placed, placed_of_chunk, tails, n_tails,
                                                                           n_pages, results, pool, out);
    return cudaGetLastError();
  }
  const uint32_t tail_ctas = (n_tails * kTailUnits + kResolveWarps - 1) / kResolveWarps;
  resolve_kernel<kResolveTails><<<tail_ctas, kResolveThreads, 0, stream>>>(placed, placed_of_chunk, tails, n_tails,
                                                                           n_pages, results, pool, out);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(body_ctas);
  cfg.blockDim = dim3(kResolveThreads);
  cfg.stream = stream;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, resolve_kernel<kResolveBodies>, placed, placed_of_chunk, tails, n_tails, n_pages,
                            results, pool, out);
}

cudaError_t launch_crc(const CrcBlock* blocks, uint32_t n_blocks, const uint8_t* out,
                       const uint64_t* mem_end, uint32_t* mem_raw, const uint64_t* mem_trailer,
                       const uint64_t* mem_len, uint32_t n_mem, const uint8_t* in,
                       int32_t* mem_status, int sms, cudaStream_t stream) {
  if (n_blocks) {
    const uint32_t cap = (uint32_t)sms * kCrcCtasPerSm;
    const uint32_t grid = n_blocks < cap ? n_blocks : cap;
    crc_blocks_kernel<<<grid, kCrcThreads, kCrcSmem, stream>>>(blocks, n_blocks, out, mem_raw);
  }
  if (n_mem)
    member_check_kernel<<<(n_mem + 7) / 8, 256, 0, stream>>>(mem_trailer, mem_len, mem_end, n_mem, in,
                                                            mem_raw, mem_status);
  return cudaGetLastError();
}

}  // namespace gzgpu
