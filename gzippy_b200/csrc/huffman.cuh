// huffman.cuh -- code tables, the warp bit reader and the block header parse
// (RFC 1951), shared by the inflate kernels and the sync-start search.
#pragma once
#include <cstdint>

#include "common.cuh"
#include "inflate.cuh"

namespace gzgpu {

__constant__ uint16_t c_len_base[29] = {3,  4,  5,  6,  7,  8,  9,  10,  11,  13,
                                        15, 17, 19, 23, 27, 31, 35, 43,  51,  59,
                                        67, 83, 99, 115, 131, 163, 195, 227, 258};
__constant__ uint8_t c_len_extra[29] = {0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 2, 2, 2,
                                        2, 3, 3, 3, 3, 4, 4, 4, 4, 5, 5, 5, 5, 0};
__constant__ uint16_t c_dist_base[32] = {1,    2,    3,    4,    5,    7,     9,     13,
                                         17,   25,   33,   49,   65,   97,    129,   193,
                                         257,  385,  513,  769,  1025, 1537,  2049,  3073,
                                         4097, 6145, 8193, 12289, 16385, 24577, 0,     0};
__constant__ uint8_t c_dist_extra[32] = {0, 0, 0, 0, 1, 1, 2,  2,  3,  3,  4,  4,  5,  5, 6, 6,
                                         7, 7, 8, 8, 9, 9, 10, 10, 11, 11, 12, 12, 13, 13, 0, 0};
__constant__ uint8_t c_cl_order[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

// litlen / dist table entry: [3:0] code length (0 = longer than the LUT or
// invalid), [7:4] extra bits, [9:8] kind, [31:16] literal / base value.
enum : uint32_t { kKindLit = 0, kKindLen = 1, kKindEob = 2, kKindBad = 3 };

__device__ __forceinline__ uint32_t litlen_entry(uint32_t sym, uint32_t L) {
  if (sym < 256) return (sym << 16) | (kKindLit << 8) | L;
  if (sym == 256) return (kKindEob << 8) | L;
  if (sym <= 285) {
    uint32_t k = sym - 257;
    return ((uint32_t)c_len_base[k] << 16) | ((uint32_t)c_len_extra[k] << 4) | (kKindLen << 8) | L;
  }
  return (kKindBad << 8) | L;
}
__device__ __forceinline__ uint32_t dist_entry(uint32_t sym, uint32_t L) {
  if (sym < 30) return ((uint32_t)c_dist_base[sym] << 16) | ((uint32_t)c_dist_extra[sym] << 4) | L;
  return (kKindBad << 8) | L;
}
__device__ __forceinline__ uint32_t pre_entry(uint32_t sym, uint32_t L) { return (sym << 16) | L; }

// A block header's working set: the precode's table, the code lengths read
// with it (literal/length codes at 0, distance codes at 288) and scratch.
struct HeaderScratch {
  uint32_t pre_lut[128];
  uint16_t pre_count[16], pre_first[16], pre_offs[16], next[16];
  uint16_t pre_sorted[20];
  uint8_t lens[320];
};

// Per-warp Huffman tables (shared memory): ring kernel and sync-start search.
template <int LB>
struct alignas(16) Tables {
  uint32_t lit_lut[1 << LB];
  uint32_t dist_lut[1 << kDistBits];
  uint16_t lit_sorted[288];
  uint16_t dist_sorted[32];
  uint16_t lit_count[16], lit_first[16], lit_offs[16];
  uint16_t dist_count[16], dist_first[16], dist_offs[16];
  HeaderScratch h;
};

// ---------------------------------------------------------------------------
// Bit reader over the register-staged input windows: a 128-bit bit window
// (bb = bits 0..63, hi = bits 64..127), refilled to > 96 valid bits.
// ---------------------------------------------------------------------------
struct BitReader {
  const uint32_t* in32;
  uint64_t win_base;  // word index of the current input window
  uint32_t win_cur;   // this lane's word of the current input window
  uint32_t win_next;  // this lane's word of the next input window
  uint64_t bb, hi;    // bit window (LSB = next bit)
  int bc;             // valid bits in the window
  uint64_t wpos;      // word index of the next word to append
  uint64_t limit_words;

  __device__ __forceinline__ void load_windows(uint64_t base, int lane) {
    win_base = base;
    win_cur = in32[base + lane];
    win_next = in32[base + 32 + lane];
  }
  __device__ __forceinline__ uint32_t word(uint64_t wi, int lane) {
    uint64_t rel = wi - win_base;
    if (rel >= 32) {
      if (rel < 64) {
        win_base += 32;
        win_cur = win_next;
        win_next = in32[win_base + 32 + lane];
      } else {
        load_windows(wi & ~31ull, lane);
      }
      rel = wi - win_base;
    }
    return __shfl_sync(0xFFFFFFFFu, win_cur, (int)rel);
  }
  __device__ __forceinline__ void seek(uint64_t bit, int lane) {
    uint64_t wi = bit >> 5;
    if (wi < win_base || wi >= win_base + 32) load_windows(wi & ~31ull, lane);
    bb = word(wi, lane) >> (bit & 31);
    hi = 0;
    bc = 32 - (int)(bit & 31);
    wpos = wi + 1;
  }
  __device__ __forceinline__ void append(uint32_t w) {
    if (bc < 64) {
      bb |= (uint64_t)w << bc;
      if (bc > 32) hi |= (uint64_t)w >> (64 - bc);
    } else {
      hi |= (uint64_t)w << (bc - 64);
    }
    bc += 32;
  }
  __device__ __forceinline__ void refill(int lane) {
    while (bc <= 96) append(word(wpos++, lane));
  }
  __device__ __forceinline__ void consume(int k) {  // 0 <= k < 64
    if (k) {
      bb = (bb >> k) | (hi << (64 - k));
      hi >>= k;
      bc -= k;
    }
  }
  __device__ __forceinline__ uint64_t pos() const { return wpos * 32 - (uint64_t)bc; }
  __device__ __forceinline__ bool overrun() const { return wpos > limit_words; }
};

// ---------------------------------------------------------------------------
// Canonical Huffman code, warp-cooperative: per-length counts, first codes
// and the symbols sorted by (length, symbol).  lens[0..n) in shared memory.
// Acceptance follows zlib: over-subscribed sets fail; incomplete sets pass
// only when the longest code is one bit or the set is empty.
// ---------------------------------------------------------------------------
static __device__ __noinline__ bool canon_build(const uint8_t* lens, int n, uint16_t* count,
                                                uint16_t* first, uint16_t* offs, uint16_t* sorted,
                                                uint16_t* next, int lane) {
  // histogram by ballots: lane L (1..15) accumulates count[L]
  uint32_t cnt_l = 0;
  for (int g = 0; g < n; g += 32) {
    int s = g + lane;
    uint32_t l = s < n ? lens[s] : 0;
#pragma unroll
    for (int L = 1; L <= 15; L++) {
      uint32_t m = __ballot_sync(0xFFFFFFFFu, l == (uint32_t)L);
      if (lane == L) cnt_l += __popc(m);
    }
  }
  if (lane >= 1 && lane <= 15) count[lane] = (uint16_t)cnt_l;
  if (lane == 0) count[0] = 0;
  __syncwarp();
  // first code / offsets, validity (every lane computes the same values)
  int left = 1, maxl = 0;
  uint32_t code = 0, off = 0;
  for (int L = 1; L <= 15; L++) {
    uint32_t c = count[L];
    left = (left << 1) - (int)c;
    if (c) maxl = L;
    if (L > 1) code = (code + count[L - 1]) << 1;
    if (lane == L) {
      first[L] = (uint16_t)code;
      offs[L] = (uint16_t)off;
      next[L] = (uint16_t)off;
    }
    off += c;
    if (left < 0) break;
  }
  bool ok = left >= 0 && !(maxl > 0 && left > 0 && maxl != 1);
  __syncwarp();
  if (!ok) return false;
  // symbols sorted by (length, symbol)
  for (int g = 0; g < n; g += 32) {
    int s = g + lane;
    uint32_t l = s < n ? lens[s] : 0;
    uint32_t peers = __match_any_sync(0xFFFFFFFFu, l);
    uint32_t rank = __popc(peers & ((1u << lane) - 1));
    if (l) sorted[next[l] + rank] = (uint16_t)s;
    __syncwarp();
    if (l && (__ffs(peers) - 1) == lane) next[l] = (uint16_t)(next[l] + __popc(peers));
    __syncwarp();
  }
  return true;
}

// Primary LUT entry i of a canonical code: the entry of the code whose bits
// (LSB-first) are the low bits of i; 0 when the code is longer than TB bits
// or unused.
template <int TB, typename EntryFn>
__device__ __forceinline__ uint32_t lut_entry(uint32_t i, const uint16_t* count, const uint16_t* first,
                                              const uint16_t* offs, const uint16_t* sorted,
                                              EntryFn entry) {
  const uint32_t rev = __brev(i) >> (32 - TB);  // MSB-first code bits
  for (int L = 1; L <= TB; L++) {
    const uint32_t idx = (rev >> (TB - L)) - first[L];
    if (idx < count[L]) return entry(sorted[offs[L] + idx], (uint32_t)L);
  }
  return 0;
}

template <int TB, typename EntryFn>
__device__ bool build_table(const uint8_t* lens, int n, uint16_t* count, uint16_t* first,
                            uint16_t* offs, uint16_t* sorted, uint16_t* next, uint32_t* lut,
                            int lane, EntryFn entry) {
  if (!canon_build(lens, n, count, first, offs, sorted, next, lane)) return false;
  for (int i = lane; i < (1 << TB); i += 32)
    lut[i] = lut_entry<TB>((uint32_t)i, count, first, offs, sorted, entry);
  __syncwarp();
  return true;
}

// Codes longer than the LUT: canonical first-code search on 15 bits.
// Returns the entry, or 0 for an invalid code.
template <int TB, typename EntryFn>
__device__ __forceinline__ uint32_t slow_decode(uint64_t bb, const uint16_t* count,
                                                const uint16_t* first, const uint16_t* offs,
                                                const uint16_t* sorted, EntryFn entry) {
  uint32_t rev = __brev((uint32_t)bb) >> 17;  // 15 code bits, first bit = MSB
  for (int L = TB + 1; L <= 15; L++) {
    uint32_t c = rev >> (15 - L);
    uint32_t idx = c - first[L];
    if (idx < count[L]) return entry(sorted[offs[L] + idx], (uint32_t)L);
  }
  return 0;
}

// Code lengths of a fixed (btype 1) or dynamic (btype 2) block into
// h->lens; the 3 header bits are already consumed.  One warp.  Returns kOk or
// an error status; nlen / ndist = number of literal/length and distance codes.
static __device__ __noinline__ int32_t read_lens(BitReader& br, uint32_t btype, HeaderScratch* h,
                                                 uint64_t trunc_words, int lane, int& nlen,
                                                 int& ndist) {
  bool ok;
  if (btype == 1) {
    // fixed Huffman (RFC 1951 3.2.6): litlen 0..287, then 32 distance codes
    for (int s = lane; s < 320; s += 32) {
      uint8_t l;
      if (s < 144) l = 8;
      else if (s < 256) l = 9;
      else if (s < 280) l = 7;
      else if (s < 288) l = 8;
      else l = 5;
      h->lens[s] = l;
    }
    __syncwarp();
    nlen = 288;
    ndist = 32;
    return kOk;
  }
  // dynamic header (RFC 1951 3.2.7)
  br.refill(lane);
  const uint32_t hdr = (uint32_t)br.bb & 0x3FFF;
  br.consume(14);
  nlen = 257 + (hdr & 31);
  ndist = 1 + ((hdr >> 5) & 31);
  const int ncl = 4 + (hdr >> 10);
  if (nlen > 286 || ndist > 30) return kBadDeflate;
  // code-length code lengths: 3 bits each, read as up to 10 + 9
  uint32_t clv = 0;
  int n1 = ncl < 10 ? ncl : 10;
  br.refill(lane);
  if (lane < n1) clv = (uint32_t)(br.bb >> (3 * lane)) & 7;
  br.consume(3 * n1);
  br.refill(lane);
  if (lane >= 10 && lane < ncl) clv = (uint32_t)(br.bb >> (3 * (lane - 10))) & 7;
  br.consume(3 * (ncl - n1));
  if (lane < 19) h->lens[296 + c_cl_order[lane]] = (uint8_t)clv;
  __syncwarp();
  ok = build_table<7>(h->lens + 296, 19, h->pre_count, h->pre_first, h->pre_offs, h->pre_sorted,
                      h->next, h->pre_lut, lane, pre_entry);
  if (!ok) return kBadDeflate;
  int i = 0, total = nlen + ndist;
  uint32_t prev = 0;
  while (i < total) {
    br.refill(lane);
    if (br.overrun()) {
      ok = false;
      break;
    }
    uint32_t e = h->pre_lut[br.bb & 127];
    uint32_t L = e & 15;
    if (L == 0) {
      ok = false;
      break;
    }
    uint32_t sym = e >> 16;
    br.consume(L);
    if (sym < 16) {
      if (lane == 0) h->lens[i] = (uint8_t)sym;
      prev = sym;
      i++;
      continue;
    }
    int rep;
    uint32_t v = 0;
    if (sym == 16) {
      if (i == 0) {
        ok = false;
        break;
      }
      v = prev;
      rep = 3 + (int)(br.bb & 3);
      br.consume(2);
    } else if (sym == 17) {
      rep = 3 + (int)(br.bb & 7);
      br.consume(3);
    } else {
      rep = 11 + (int)(br.bb & 127);
      br.consume(7);
    }
    if (i + rep > total) {
      ok = false;
      break;
    }
    for (int j = lane; j < rep; j += 32) h->lens[i + j] = (uint8_t)v;
    prev = v;
    i += rep;
  }
  __syncwarp();
  if (br.overrun()) return br.wpos > trunc_words ? kTruncated : kOvershoot;
  if (!ok || h->lens[256] == 0) return kBadDeflate;
  // the dist lengths must not alias the precode area: move them to 288+
  uint8_t dl = lane < ndist ? h->lens[nlen + lane] : 0;
  __syncwarp();
  h->lens[288 + lane] = lane < ndist ? dl : 0;
  __syncwarp();
  return kOk;
}

// read_lens and both code tables, by one warp.
template <int LB>
__device__ int32_t read_tables(BitReader& br, uint32_t btype, Tables<LB>* T, uint64_t trunc_words,
                               int lane) {
  int nlen, ndist;
  const int32_t st = read_lens(br, btype, &T->h, trunc_words, lane, nlen, ndist);
  if (st != kOk) return st;
  bool ok = build_table<LB>(T->h.lens, nlen, T->lit_count, T->lit_first, T->lit_offs, T->lit_sorted,
                            T->h.next, T->lit_lut, lane, litlen_entry);
  ok = ok && build_table<kDistBits>(T->h.lens + 288, ndist, T->dist_count, T->dist_first,
                                    T->dist_offs, T->dist_sorted, T->h.next, T->dist_lut, lane,
                                    dist_entry);
  return ok ? kOk : kBadDeflate;
}

// ---------------------------------------------------------------------------
// Page allocation (both layouts).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t alloc_page(const PagePool& pool, uint32_t cid, uint32_t gen,
                                               uint32_t seq, int lane) {
  uint32_t p = 0;
  if (lane == 0) {
    p = atomicAdd(pool.next, 1u);
    if (p < pool.cap) {
      pool.owner[p] = cid;
      pool.seq[p] = (gen << kGenShift) | seq;
    }
  }
  p = __shfl_sync(0xFFFFFFFFu, p, 0);
  return p < pool.cap ? p : kNoPage;
}

}  // namespace gzgpu
