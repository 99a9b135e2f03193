// finder.cu -- deflate block-boundary finder (K1) and chunk linking.
//
// Each speculative chunk's range [guess_bit, limit_bit) is searched for its first
// block-start candidate (predicate in finder_core.cuh): stored blocks, then sync
// starts in fixed blocks by a CTA per range, then dynamic headers by the warps of
// a grid, a segment of a range each.
#include <cstdint>

#include "barrier.cuh"
#include "common.cuh"
#include "finder.cuh"
#include "finder_core.cuh"

namespace gzgpu {

// Stored block starts, searched first for every speculative chunk: the first
// one (by byte offset, hence by start bit) in [guess_bit, limit_bit) whose
// successor passes stored_successor becomes the chunk's start, and the
// sync search and the block finder skip the chunk.  The successor check is
// a heuristic: a false start needs two LEN/NLEN matches in a row, or a
// LEN/NLEN match and a valid dynamic header, which is rare but possible.
// Correctness does not rest on it: a false start only decodes garbage that
// no predecessor hands over to, and the host chain walk repairs past it.
// The pass runs before the sync search because the raw bytes of stored
// blocks (text, runs) walk as fixed-Huffman codes and would give false sync
// starts.  One CTA of kStoredThreads per chunk; a thread screens 16 aligned
// byte offsets a round with word operations (a round covers 4 KiB, so a 24 KiB
// partition is six load latencies; offset by offset, 1 KiB a round, took
// 41 us for the 1,365 partitions of a 23 MB stream).  A dynamic header after a
// candidate's block is read by the whole warp: by one thread it is 90,000
// cycles, which the last CTAs waited for (3,286 partitions of a mixed stream:
// 89 us, now 49).
constexpr int kStoredThreads = 256;

// A warp's scratch for dyn_candidate_warp
struct HeaderTest {
  uint8_t sorted[32];  // the precode's symbols in code order
  uint8_t lut[128];    // and its table, entry: symbol | length << 5
};
__device__ __noinline__ bool dyn_candidate_warp(const uint8_t* in, uint64_t nbytes, uint64_t bit,
                                                HeaderTest& W, int lane, uint32_t& mean);

__global__ void __launch_bounds__(kStoredThreads)
    stored_kernel(const uint8_t* __restrict__ in, ChunkDesc* descs,
                  const uint32_t* __restrict__ spec, uint32_t n_spec, unsigned long long* best) {
  __shared__ unsigned long long s_first;
  __shared__ HeaderTest ht[kStoredThreads / 32];
  if (blockIdx.x >= n_spec) return;
  if (threadIdx.x == 0) best[blockIdx.x] = ~0ull;  // for find_kernel
  ChunkDesc& d = descs[spec[blockIdx.x]];
  if (d.flags & kChunkValid) return;
  const uint64_t from = d.guess_bit, to = d.limit_bit, nbytes = d.in_end;
  if (threadIdx.x == 0) s_first = ~0ull;
  cta_sync();
  const uint64_t begin = max((from + 3 + 7) / 8, (uint64_t)2);
  const uint64_t until = nbytes >= 5 ? min((to + 7) / 8, nbytes - 4) : 0;
  // (the next round's bytes are on their way while this one's are tested)
  uint64_t ob = (begin & ~15ull) + 16 * (uint64_t)threadIdx.x;
  uint4 v = make_uint4(0, 0, 0, 0);
  uint32_t v4 = 0;
  auto load = [&]() {
    if (ob >= until) return;
    v = *reinterpret_cast<const uint4*>(in + ob);
    v4 = *reinterpret_cast<const uint32_t*>(in + ob + 16);
  };
  load();
  for (uint64_t base = begin & ~15ull; base < until; base += 16 * kStoredThreads) {
    const uint32_t w[5] = {v.x, v.y, v.z, v.w, v4};
    const uint64_t at = ob;
    ob += 16 * kStoredThreads;
    load();
    uint32_t m = 0;
    if (at < until) {
#pragma unroll
      for (int k = 0; k < 16; k++) {
        const uint32_t sz = __funnelshift_r(w[k >> 2], w[(k >> 2) + 1 < 5 ? (k >> 2) + 1 : 4], 8 * (k & 3));
        m |= (((sz ^ (sz >> 16)) & 0xFFFFu) == 0xFFFFu ? 1u : 0u) << k;
      }
      if (at < begin) m &= 0xFFFFFFFFu << (begin - at);
      if (at + 16 > until) m &= (1u << (until - at)) - 1;
    }
    bool found = false;
    for (;;) {
      // this lane's next candidate whose successor's header decides
      uint64_t off = 0, hdr = 0;
      while (m && !hdr) {
        off = at + (uint64_t)(__ffs(m) - 1);
        m &= m - 1;
        uint64_t lo = 0, hi = 0;
        if (!stored_candidate(in, nbytes, off, from, to, to, lo, hi)) continue;
        const uint64_t next = off + 4 + (in[off] | (in[off + 1] << 8));
        const int s = stored_successor(in, nbytes, next);
        if (s == kSuccHeader) hdr = next * 8;
        if (s == kSuccYes) {
          atomicMin(&s_first, (unsigned long long)off);
          found = true;
          m = 0;
        }
      }
      __syncwarp();
      uint32_t b = __ballot_sync(0xFFFFFFFFu, hdr != 0);
      if (!b) break;
      for (; b; b &= b - 1) {
        const int src = __ffs(b) - 1;
        uint32_t mean;
        const bool ok = dyn_candidate_warp(in, nbytes, __shfl_sync(0xFFFFFFFFu, hdr, src),
                                           ht[threadIdx.x >> 5], threadIdx.x & 31, mean);
        if (ok && (int)(threadIdx.x & 31) == src) {
          atomicMin(&s_first, (unsigned long long)off);
          found = true;
          m = 0;
        }
        __syncwarp();
      }
    }
    if (cta_sync_or(found)) break;
  }
  if (threadIdx.x == 0 && s_first != ~0ull) {
    uint64_t lo = 0, hi = 0;
    stored_candidate(in, nbytes, s_first, from, to, to, lo, hi);
    d.lo_bit = lo;
    d.start_bit = hi;
    d.flags |= kChunkValid;
    d.est_ratio = 1.f;
  }
}

// The precode leaf count of 4 code-length codes (12 bits) for every value,
// built at compile time; each CTA copies it to shared memory.
struct LeafLut {
  uint16_t v[4096];
  constexpr LeafLut() : v() {
    for (int i = 0; i < 4096; i++) {
      uint32_t sum = 0;
      for (int k = 0; k < 4; k++) {
        const uint32_t L = (i >> (3 * k)) & 7;
        sum += L ? 1u << (7 - L) : 0u;
      }
      v[i] = (uint16_t)sum;
    }
  }
};
__device__ const LeafLut d_leaf_lut = LeafLut();

// Dynamic headers.  The ranges still without a start are searched in segments
// of up to kFindSeg bits, one warp per segment, segment 0 of every range first, then
// segment 1, and so on: a range's later segments are skipped once an earlier
// one has a hit, while a small job's segments all run at once.  (One CTA per
// range, walking it from its start, took 370 us for the 30 ranges of a 1 MB
// stream and 630 us for 1,365 ranges, mostly latency.)  A segment's words go
// to shared memory; its bit offsets are screened in passes of 4096: the
// 13-bit filter for 32 offsets per lane at once, the survivors (1 in 9) to a
// list, the precode leaf count for 32 of them at a time; what is left
// (about 1 in 100 of the list, in order) gets the full header test.
constexpr int kFindWarps = 8;
constexpr uint32_t kFindSeg = 8192;                // bits per segment, at most
constexpr uint32_t kFindSegMin = 1024;             // and at least
constexpr uint32_t kFindPass = 4096;               // bits per screening pass
// most survivors of a pass: three bits apart (BFINAL 0, BTYPE 10); near a
// member's end, where BFINAL may be either, two, in passes half as long
constexpr uint32_t kFindList = kFindPass / 3 + 2;
static_assert(kFindPass / 4 + 2 <= kFindList, "");
constexpr uint32_t kFindFull = 64;                 // full tests held
// a hit: its bit, then its code's mean bytes per symbol in eighths (up to 258)
constexpr int kMeanBits = 12;

struct FindWarp {
  uint32_t w[kFindSeg / 32 + 6];
  uint16_t list[kFindList];
  uint16_t full[kFindFull];
  HeaderTest ht;
  uint32_t n_full;
};

// dyn_candidate_full (finder_core.cuh) by a whole warp, for one candidate.
// Every lane decodes the code length that would start at its bit of the next
// 32; a walk over shuffles picks the real ones (about nine), which are then
// weighed together.  A true header is 200 and more lengths one after another,
// 90,000 cycles and more for a thread by itself, 15,000 so; a false one ends
// within two or three such steps.  mean: of a true one, the bytes a symbol
// gives on average by its code (a code of length v stands for a probability of
// 2^-v), in units of 2^-15.
__device__ __noinline__ bool dyn_candidate_warp(const uint8_t* in, uint64_t nbytes, uint64_t bit,
                                                HeaderTest& W, int lane, uint32_t& mean) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint32_t below = (1u << lane) - 1;
  const uint32_t h = (uint32_t)peek_bits(in, nbytes, bit, 17);
  const uint32_t hl = 257 + ((h >> 3) & 31), total = hl + 1 + ((h >> 8) & 31);
  const int pc = (int)((h >> 13) & 15) + 4;
  const uint64_t pos0 = bit + 17 + 3 * pc;  // first bit of the code lengths
  uint64_t wbase = pos0 >> 5;
  uint32_t word = in32[wbase + lane], word2 = in32[wbase + 32 + lane];  // 2048 bits from there on
  // the precode, canonical: lane s has symbol s
  const uint64_t pbits = peek_bits(in, nbytes, bit + 17, 3 * pc);
  const int place = lane < 16 ? (lane == 0 ? 3 : (lane < 8 ? 19 - 2 * lane : 2 * lane - 12)) : lane - 16;
  const uint32_t my = lane < 19 ? (uint32_t)(pbits >> (3 * place)) & 7 : 0u;
  uint32_t lim[8], base[8];
  {
    uint32_t code = 0, off = 0, c = 0, leaves = 0, at = 0;
#pragma unroll
    for (uint32_t l = 1; l < 8; l++) {
      const uint32_t b = __ballot_sync(kAll, my == l);
      code = (code + c) << 1;
      c = __popc(b);
      lim[l] = (code + c) << (7 - l);
      base[l] = off - code;
      if (my == l) at = off + __popc(b & below);
      off += c;
      leaves += c << (15 - l);
    }
    const uint32_t longer = __ballot_sync(kAll, my > 1);
    if (!kraft_exact(leaves, longer)) return false;
    if (my) W.sorted[at] = (uint8_t)lane;
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t rev = __brev(lane + 32 * k) >> 25;
    uint32_t L = 1, b = base[1];
#pragma unroll
    for (int l = 1; l < 7; l++)
      if (rev >= lim[l]) {
        L = l + 1;
        b = base[l + 1];
      }
    W.lut[lane + 32 * k] = rev >= lim[7] ? (uint8_t)0 : (uint8_t)(W.sorted[(rev >> (7 - L)) + b] | L << 5);
  }
  __syncwarp();
  const uint64_t nbits = nbytes * 8;
  const uint32_t room = pos0 < nbits ? (uint32_t)min(nbits - pos0, (uint64_t)1 << 20) : 0u;
  uint32_t rel = (uint32_t)(pos0 & 31);  // position, from wbase on
  uint32_t rel0 = rel;
  uint32_t n = 0, prev = 0;              // lengths read, the last of them
  mean = 1u << 15;
  uint32_t lit = 0, dist = 0, lit_gt1 = 0, dist_gt1 = 0, eob = 0;
  while (n < total) {
    if (rel >= 1024 + 960) {  // (rare: a header of over 2,000 bits)
      word = word2;
      wbase += 32;
      word2 = in32[wbase + 32 + lane];
      rel -= 1024;
      rel0 -= 1024;  // only the difference counts
    }
    const uint32_t j = rel >> 5, t = (rel & 31) + lane;
    const uint32_t wa = __shfl_sync(kAll, j < 32 ? word : word2, j & 31);
    const uint32_t wb = __shfl_sync(kAll, j + 1 < 32 ? word : word2, (j + 1) & 31);
    const uint32_t wc = __shfl_sync(kAll, j + 2 < 32 ? word : word2, (j + 2) & 31);
    const uint32_t x = __funnelshift_r(t < 32 ? wa : wb, t < 32 ? wb : wc, t & 31);
    const uint32_t e = W.lut[x & 127], L = e >> 5, sym = e & 31;
    const uint32_t xb = sym < 16 ? 0u : (sym == 16 ? 2u : (sym == 17 ? 3u : 7u));
    const uint32_t rep = sym < 16 ? 1u : ((x >> L) & ((1u << xb) - 1)) + (sym == 18 ? 11u : 3u);
    // next length's bit (0x40: no such code), and the one after that
    const uint32_t nx = L ? lane + L + xb : 0x40u;
    const uint32_t nx2 = __shfl_sync(kAll, nx, nx & 31);
    const uint32_t hop = nx | (nx < 32 ? nx2 : 0xFFu) << 8;
    uint32_t chain = 0, p = 0;
    for (;;) {
      const uint32_t v = __shfl_sync(kAll, hop, p), a = v & 0xFF, b = v >> 8;
      if (a == 0x40) break;  // not a code at p
      chain |= 1u << p;
      if (a >= 32) {
        p = a;
        break;
      }
      if (b == 0x40) {  // not a code at a
        p = a;
        break;
      }
      chain |= 1u << a;
      p = b;
      if (p >= 32) break;
    }
    const bool ends = p < 32;  // the chain runs into an invalid code at p
    const bool on = (chain >> lane) & 1;
    // a repeat of the one before (16) takes the value of the last other symbol
    const uint32_t own = __ballot_sync(kAll, on && sym != 16);
    const uint32_t before = own & (below | 1u << lane);
    const uint32_t v0 = __shfl_sync(kAll, sym < 16 ? sym : 0u, 31 - __clz(before | 1u));
    const uint32_t v = before ? v0 : prev;
    const uint32_t r = on ? rep : 0u;
    uint32_t at = r;  // lengths up to and with this one
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(kAll, at, d);
      if (lane >= d) at += u;
    }
    const uint32_t i = n + at - r;                 // this one's place
    const bool use = on && i < total;
    // bad: a repeat with nothing before it, past the last length, past the input
    const bool bad = use && ((sym == 16 && i == 0) || i + r > total || rel - rel0 + lane + L + xb > room);
    const uint32_t n_lit = use && i < hl ? min(r, hl - i) : 0u, n_dist = use ? r - n_lit : 0u;
    if (__any_sync(kAll, bad)) return false;
    lit += __reduce_add_sync(kAll, v ? n_lit << (15 - v) : 0u);
    dist += __reduce_add_sync(kAll, v ? n_dist << (15 - v) : 0u);
    // Kraft sums only grow: an over-subscribed set fails the final test
    if (lit > (1u << 15) || dist > (1u << 15)) return false;
    lit_gt1 |= __ballot_sync(kAll, v > 1 && n_lit);
    dist_gt1 |= __ballot_sync(kAll, v > 1 && n_dist);
    eob |= __ballot_sync(kAll, use && v && i <= 256 && 256 < i + r);
    {
      // length symbols: more than a byte each (a repeat's by the first of them)
      const uint32_t s = max(i, 257u);
      const uint32_t c = v && i + n_lit > s ? i + n_lit - s : 0u;
      const uint32_t more = c ? f_len_base[min(s - 257, 28u)] + (1u << f_len_extra[min(s - 257, 28u)]) / 2 - 1 : 0u;
      mean += __reduce_add_sync(kAll, c * more << (15 - v));
    }
    const uint32_t last = 31 - __clz(chain | 1u);
    n += __shfl_sync(kAll, at, 31);
    prev = __shfl_sync(kAll, v, last);
    if (ends && n < total) return false;
    rel += p;
  }
  return eob && kraft_exact(lit, lit_gt1) && kraft_exact(dist, dist_gt1);
}

__global__ void __launch_bounds__(32 * kFindWarps)
    find_kernel(const uint8_t* __restrict__ in, const ChunkDesc* __restrict__ descs,
                const uint32_t* __restrict__ spec, uint32_t n_spec, uint32_t n_seg, uint32_t seg,
                unsigned long long* best, uint32_t* next_item) {
  __shared__ uint16_t leaf[4096];
  __shared__ FindWarp fw[kFindWarps];
  const int lane = threadIdx.x & 31;
  FindWarp& W = fw[threadIdx.x >> 5];
  for (uint32_t i = threadIdx.x; i < 4096 / 8; i += 32 * kFindWarps)
    reinterpret_cast<uint4*>(leaf)[i] = reinterpret_cast<const uint4*>(d_leaf_lut.v)[i];
  cta_sync();
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint64_t n_items = (uint64_t)n_spec * n_seg;
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(next_item, 1u);
    item = __shfl_sync(0xFFFFFFFFu, item, 0);
    if (item >= n_items) break;
    const uint32_t k = item % n_spec, sg = item / n_spec;
    const ChunkDesc& d = descs[spec[k]];
    if (d.flags & kChunkValid) continue;  // a stored or sync start was found first
    const uint64_t nbytes = d.in_end, nbits = nbytes * 8;
    const uint64_t from = d.guess_bit, to = min(d.limit_bit, nbits);
    // segments are cut at word boundaries of the input
    const uint64_t s0 = (from & ~31ull) + (uint64_t)sg * seg;
    if (s0 >= to) continue;
    if (*(volatile unsigned long long*)&best[k] >> kMeanBits < s0) continue;
    const uint32_t len = (uint32_t)min((uint64_t)seg, to - s0);
    const uint32_t first = from > s0 ? (uint32_t)(from - s0) : 0u;
    // the segment's words, and the 81 bits after it (a header up to its precode)
    __syncwarp();
    const uint64_t wi = s0 >> 5;
#pragma unroll
    for (uint32_t j = 0; j < kFindSeg / 32 + 6; j += 32)
      if (j + lane < kFindSeg / 32 + 6 && 32 * (j + lane) < len + 160) W.w[j + lane] = in32[wi + j + lane];
    if (lane == 0) W.n_full = 0;
    __syncwarp();
    uint32_t hit = kFindSeg, mean = 0;  // lowest passing offset, its code's bytes per symbol
    const bool tail = d.flags & kChunkTail;
    const uint32_t pass = tail ? kFindPass / 2 : kFindPass;
    for (uint32_t p0 = 0; p0 < len && hit == kFindSeg; p0 += pass) {
      const uint32_t p1 = min(len, p0 + pass);
      uint32_t m[kFindPass / 1024], c = 0;
#pragma unroll
      for (uint32_t q = 0; q < kFindPass / 1024; q++) {
        const uint32_t p = p0 + 1024 * q + 32 * lane;
        uint32_t v = 0;
        if (p < p1) {
          v = dyn_filter32((uint64_t)W.w[(p >> 5) + 1] << 32 | W.w[p >> 5], tail);
          if (p + 32 > p1) v &= (1u << (p1 - p)) - 1;
          if (p < first) v &= p + 32 > first ? 0xFFFFFFFFu << (first - p) : 0u;
        }
        m[q] = v;
        c += __popc(v);
      }
      uint32_t at = c;
#pragma unroll
      for (int b = 1; b < 32; b <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, at, b);
        if (lane >= b) at += v;
      }
      const uint32_t tot = __shfl_sync(0xFFFFFFFFu, at, 31);
      at -= c;
#pragma unroll
      for (uint32_t q = 0; q < kFindPass / 1024; q++)
        while (m[q]) {
          W.list[at++] = (uint16_t)(p0 + 1024 * q + 32 * lane + __ffs(m[q]) - 1);
          m[q] &= m[q] - 1;
        }
      __syncwarp();
      for (uint32_t j0 = 0; j0 < tot; j0 += 32) {
        const bool act = j0 + lane < tot;
        const uint32_t p = act ? W.list[j0 + lane] : 0u;
        // HCLEN and the precode: bits 13 .. 76 of the header
        const uint32_t a = (p + 13) >> 5, sh = (p + 13) & 31;
        const uint32_t w1 = W.w[a + 1];
        const uint32_t lo = __funnelshift_r(W.w[a], w1, sh), hi = __funnelshift_r(w1, W.w[a + 2], sh);
        const uint32_t n = 3 * ((lo & 15) + 4);  // precode bits
        uint64_t pb = ((uint64_t)hi << 32 | lo) >> 4;
        pb &= (1ull << n) - 1;
        const uint32_t x0 = (uint32_t)pb, x1 = (uint32_t)(pb >> 24);
        const uint32_t sum = leaf[x0 & 0xFFF] + leaf[(x0 >> 12) & 0xFFF] + leaf[x1 & 0xFFF] +
                             leaf[(x1 >> 12) & 0xFFF] + leaf[(uint32_t)(pb >> 48)];
        // a complete code, or a single code of one bit
        const bool ok = act && (sum == 128 || (sum == 64 && !(pb & (pb - 1)))) && s0 + p + 17 + n <= nbits;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, ok);
        if (!b) continue;
        uint32_t n0 = W.n_full;
        __syncwarp();
        if (n0 + __popc(b) > kFindFull) {
          // (rare) the held ones first
          for (uint32_t j = 0; j < n0 && hit == kFindSeg; j++)
            if (dyn_candidate_warp(in, nbytes, s0 + W.full[j], W.ht, lane, mean)) hit = W.full[j];
          __syncwarp();
          n0 = 0;
        }
        if (ok) W.full[n0 + __popc(b & ((1u << lane) - 1))] = (uint16_t)p;
        if (lane == 0) W.n_full = n0 + __popc(b);
        __syncwarp();
      }
      const uint32_t n0 = W.n_full;
      for (uint32_t j = 0; j < n0 && hit == kFindSeg; j++)
        if (dyn_candidate_warp(in, nbytes, s0 + W.full[j], W.ht, lane, mean)) hit = W.full[j];
      __syncwarp();
      if (lane == 0) W.n_full = 0;
      __syncwarp();
    }
    if (hit < kFindSeg && lane == 0)
      atomicMin(&best[k], (unsigned long long)(s0 + hit) << kMeanBits | min(mean >> 12, (1u << kMeanBits) - 1));
  }
}

// the dynamic starts found, into the chunk table; ratio: with the output
// estimate of their headers
__global__ void assign_kernel(const uint8_t* __restrict__ in, ChunkDesc* descs,
                              const uint32_t* __restrict__ spec, uint32_t n_spec,
                              const unsigned long long* __restrict__ best, int ratio,
                              uint32_t* next_item) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) *next_item = 0;
  if (k >= n_spec) return;
  ChunkDesc& d = descs[spec[k]];
  if ((d.flags & kChunkValid) || best[k] == ~0ull) return;
  d.lo_bit = d.start_bit = best[k] >> kMeanBits;
  d.flags |= kChunkValid;
  // (without the codes' lengths: a symbol taken for two bytes)
  d.est_ratio = ratio ? dyn_header_ratio(in, d.in_end, d.start_bit)
                      : (float)(best[k] & ((1u << kMeanBits) - 1)) * (0.125f / 2);
}

// Sync starts in fixed-Huffman data (finder_core.cuh), searched for every
// speculative chunk before the block finder, which then skips the chunks that
// have one.  One CTA of kSyncOffsets threads per chunk, each walking the fixed
// code's symbols from one start bit; the walk must end inside the chunk's range
// and the input.  Walks go on in steps of kSyncStep bits and stop as soon as
// fewer than two are left (other data fails within a few hundred symbols);
// 1,365 ranges of text took 100 us when every walk ran to its end and one
// thread compared the ends.
constexpr uint32_t kSyncStep = 512;

__global__ void __launch_bounds__(kSyncOffsets)
    sync_kernel(const uint8_t* __restrict__ in, ChunkDesc* descs, const uint32_t* __restrict__ spec,
                uint32_t n_spec, uint32_t* n_sync) {
  constexpr uint32_t kWords = sync_words(kSyncOffsets, kSyncSpan);
  __shared__ uint32_t sw[kWords];
  __shared__ uint8_t lut[512], dlut[32];
  __shared__ uint32_t ends[kSyncOffsets];
  __shared__ unsigned long long top;
  if (blockIdx.x >= n_spec) return;
  ChunkDesc& d = descs[spec[blockIdx.x]];
  if (d.flags & kChunkValid) return;
  const uint64_t from = d.guess_bit, to = d.limit_bit, nbytes = d.in_end;
  const uint64_t target = from + kSyncOffsets + kSyncSpan;
  if (target + 64 > to || target + 128 > nbytes * 8) return;
  const uint32_t tid = threadIdx.x;
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in) + (from >> 5);
  for (uint32_t i = tid; i < kWords; i += kSyncOffsets) sw[i] = in32[i];
  for (uint32_t i = tid; i < 512; i += kSyncOffsets) lut[i] = (uint8_t)fixed_entry(i);
  if (tid < 32) {
    const uint32_t dc = __brev(tid) >> 27;
    dlut[tid] = dc >= 30 ? 0xFF : (uint8_t)(5 + f_dist_extra[dc]);
  }
  if (tid == 0) top = 0;
  cta_sync();
  const uint32_t rel = (uint32_t)(from & 31);  // positions below count from the word of `from`
  const uint32_t goal = rel + kSyncOffsets + (uint32_t)kSyncSpan;
  uint32_t p = rel + tid;
  bool ok = true;
  for (uint32_t step = rel + kSyncOffsets + kSyncStep;; step += kSyncStep) {
    const uint32_t e = min(step, goal);
    while (ok && p < e) {
      const uint32_t i = p >> 5;
      const uint32_t x = __funnelshift_r(sw[i], sw[i + 1], p & 31);
      const uint32_t ent = lut[x & 511];
      p += ent & 31;
      if (ent < 32) continue;  // a literal
      const uint32_t j = p >> 5;
      const uint32_t y = __funnelshift_r(sw[j], sw[j + 1], p & 31);
      if (ent >> 5 == 1) {  // a length: the distance code
        const uint32_t n = dlut[y & 31];
        ok = n != 0xFF;
        p += n;
      } else {  // EOB: another fixed block must follow
        ok = ent >> 5 == 2 && ((y >> 1) & 3) == 1;
        p += 3;
      }
    }
    if (cta_sync_count(ok) < 2) return;
    if (e == goal) break;
  }
  ends[tid] = ok ? p : 0u;
  cta_sync();
  if (ok) {
    uint32_t c = 0;
    for (uint32_t i = 0; i < kSyncOffsets; i++) c += ends[i] == p;
    // most walks first, then the lower position
    if (c >= 2) atomicMax(&top, (unsigned long long)c << 32 | (0xFFFFFFFFu - p));
  }
  cta_sync();
  if (tid == 0 && top) {
    d.lo_bit = d.start_bit = (from & ~31ull) + (0xFFFFFFFFu - (uint32_t)top);
    d.flags |= kChunkValid | kChunkSync;
    if (n_sync) atomicAdd(n_sync, 1u);
  }
}

// Decode cost of a linked chunk: its compressed bytes.  Text and noisy
// literals take the decoder 8.6 us per KB; stored data is a copy, a twentieth
// of that (only the stored blocks themselves count so: chunks that begin with
// one and go on with Huffman blocks are not short); byte runs take two to five
// times as long, so data estimated to give over twice its bytes counts half
// its output.  128 MiB mixed stream: 1.54 ms by bytes alone, 1.29 with stored
// blocks by themselves, 1.21 with the output; 600 files: 1.51 without the
// output, 1.17 with it (a file's runs went last where false sync starts made
// them look short).
__device__ float chunk_cost(const uint8_t* __restrict__ in, const ChunkDesc& d, uint64_t stop) {
  const uint64_t end = min(stop, d.in_end * 8);
  uint64_t bit = d.start_bit, copied = 0;
  if (bit >= end) return 0.f;
  const float span = (float)(end - bit) * 0.125f;
  for (int k = 0; k < 8 && bit < end && !(d.flags & kChunkSync); k++) {
    if (peek_bits(in, d.in_end, bit, 3) >> 1) break;
    const uint64_t at = (bit + 10) >> 3;  // LEN
    if (at + 2 > d.in_end) break;
    const uint64_t len = peek_bits(in, d.in_end, at * 8, 16);
    copied += len;
    bit = (at + 4 + len) * 8;
  }
  return fmaxf(span - 0.95f * (float)copied, 0.05f * span) * fmaxf(1.f, 0.5f * d.est_ratio);
}

// stop_lo of each valid chunk = lo of the next valid chunk when that one is
// speculative (member starts end their predecessor at BFINAL instead);
// valid chunks are appended to the decode work list.
// A speculative start may be a phantom whose garbage code table never fails;
// such a chunk gives up `slack` bits past its stop and the chain walk
// re-decodes the gap from the confirmed boundary instead.
__global__ void link_kernel(const uint8_t* __restrict__ in, ChunkDesc* descs, uint32_t n,
                            uint32_t* work, uint32_t* n_work, float* cost, uint64_t slack) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ChunkDesc& d = descs[i];
  if (!(d.flags & kChunkValid)) return;
  uint64_t stop = kNoStop;
  uint32_t next = kNoChunk;
  for (uint32_t j = i + 1; j < n; j++) {
    uint32_t f = descs[j].flags;
    if (descs[j].stream != d.stream) break;
    if (f & kChunkMemberFirst) {
      // a member candidate (limit_bit = its header byte): a real one follows
      // the BFINAL block, a false one lies inside this member's data
      stop = descs[j].limit_bit * 8;
      next = j;
      break;
    }
    if (f & kChunkValid) {
      stop = descs[j].lo_bit;
      next = j;
      break;
    }
  }
  d.stop_lo = stop;
  d.next = next;
  // A sync start whose table or alignment is wrong decodes garbage that a
  // complete code never rejects: it may run at most its own length (at least
  // kSyncMinSlack) past its stop.  A real one stops at its successor, or goes
  // by phantom successors mid-block to the one after (inflate.cu).
  uint64_t s = slack;
  if ((d.flags & kChunkSync) && stop != kNoStop && stop > d.start_bit)
    s = min(slack, max(stop - d.start_bit, (uint64_t)kSyncMinSlack));
  d.abort_bit = (stop != kNoStop && !(d.flags & kChunkMemberFirst)) ? stop + s : kNoStop;
  if (cost) cost[i] = chunk_cost(in, d, stop);
  else work[atomicAdd(n_work, 1u)] = i;
}

// The decode work list in descending cost (longest processing time first),
// so that the persistent decoder starts the longest chunks first and the
// short ones fill in at the end.  One CTA: a histogram over quarter-octave cost
// buckets, a scan, and a scatter (order inside a bucket is arbitrary; with
// half-octaves the decode of 600 files took 1.16 ms, so 1.08).
constexpr int kCostBuckets = 128;
__global__ void __launch_bounds__(1024)
    order_kernel(const ChunkDesc* __restrict__ descs, const float* __restrict__ cost, uint32_t n,
                 uint32_t* work, uint32_t* n_work) {
  __shared__ uint32_t hist[kCostBuckets], base[kCostBuckets];
  if (threadIdx.x < kCostBuckets) hist[threadIdx.x] = 0;
  cta_sync();
  auto bucket = [&](uint32_t i) {
    const float c = fmaxf(cost[i], 0.f) + 1.f;
    const int b = (int)(4.f * __log2f(c));
    return kCostBuckets - 1 - min(max(b, 0), kCostBuckets - 1);  // costliest first
  };
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
    if (descs[i].flags & kChunkValid) atomicAdd(&hist[bucket(i)], 1u);
  cta_sync();
  if (threadIdx.x == 0) {
    uint32_t a = 0;
    for (int b = 0; b < kCostBuckets; b++) {
      base[b] = a;
      a += hist[b];
    }
    *n_work = a;
  }
  cta_sync();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
    if (descs[i].flags & kChunkValid) work[atomicAdd(&base[bucket(i)], 1u)] = i;
}

cudaError_t launch_finder(const uint8_t* in, ChunkDesc* descs, const uint32_t* spec, uint32_t n_spec,
                          uint64_t max_bits, uint64_t* best64, uint32_t* next_item, uint32_t* n_sync,
                          bool ratio, int sms, cudaStream_t stream) {
  if (n_spec == 0) return cudaSuccess;
  // Stored starts first (a byte scan), then the fixed-code sync search: it
  // costs a fraction of a full scan, which a fixed-Huffman partition (no
  // block header to find) would need, and it fails within a few dozen
  // symbols on other data.
  unsigned long long* best = reinterpret_cast<unsigned long long*>(best64);
  stored_kernel<<<n_spec, kStoredThreads, 0, stream>>>(in, descs, spec, n_spec, best);
  sync_kernel<<<n_spec, kSyncOffsets, 0, stream>>>(in, descs, spec, n_spec, n_sync);
  // Shorter segments while a small search leaves warps without one: a segment's
  // four or five false candidates are tested one after another.  31 ranges of a
  // 1 MiB stream: 102 us in segments of 8192 bits, 42 of 1024.
  const uint64_t warps = (uint64_t)sms * 3 * kFindWarps;  // resident
  uint32_t seg = kFindSeg;
  while (seg > kFindSegMin && n_spec * ((max_bits + 31) / (seg / 2) + 1) <= warps) seg /= 2;
  const uint32_t n_seg = (uint32_t)((max_bits + 31) / seg + 1);
  const uint64_t ctas = ((uint64_t)n_spec * n_seg + kFindWarps - 1) / kFindWarps;
  const uint32_t grid = (uint32_t)(ctas < (uint64_t)sms * 4 ? ctas : (uint64_t)sms * 4);
  find_kernel<<<grid, 32 * kFindWarps, 0, stream>>>(in, descs, spec, n_spec, n_seg, seg, best,
                                                    next_item);
  assign_kernel<<<(n_spec + 127) / 128, 128, 0, stream>>>(in, descs, spec, n_spec, best, ratio,
                                                         next_item);
  return cudaGetLastError();
}

cudaError_t launch_link(const uint8_t* in, ChunkDesc* descs, uint32_t n, uint32_t* work,
                        uint32_t* n_work, float* cost, uint64_t slack_bits, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  link_kernel<<<(n + 255) / 256, 256, 0, stream>>>(in, descs, n, work, n_work, cost, slack_bits);
  if (cost) order_kernel<<<1, 1024, 0, stream>>>(descs, cost, n, work, n_work);
  return cudaGetLastError();
}

}  // namespace gzgpu
