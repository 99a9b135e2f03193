// finder_core.cuh -- block-start predicate and warp search, shared by the
// finder kernel and the inflate kernel's next-candidate retry.
//
// Predicate of the reference (src/decompress/parallel/blockfinder_validation.rs):
//   dynamic: BFINAL=0, BTYPE=10, HLIT<=29, HDIST<=29 (13-bit filter,
//            :68-150); precode leaf count 128 or 64 (validate_precode
//            :190-226) and Kraft-exact (is_valid_huffman_lengths :807-830);
//            the HLIT+257+HDIST+1 code lengths decode with the precode,
//            EOB has a code, litlen and dist sets are Kraft-exact
//            (validate_huffman_codes :836-925).  No fixed-Huffman candidates.
//   stored:  LEN == ~NLEN at a byte boundary preceded by 3 zero header bits;
//            the candidate spans [byte_bit - zero_run, byte_bit - 3]
//            (find_uncompressed_blocks :370-475).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace gzgpu {

static __constant__ uint8_t f_cl_order[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

// bits [bit, bit+k) of the input, k <= 57; bits at or past the stream end
// (byte `nbytes`) read 0.  Three aligned 32-bit loads (the buffer is padded).
static __device__ __forceinline__ uint64_t peek_bits(const uint8_t* in, uint64_t nbytes, uint64_t bit,
                                                     int k) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint64_t wi = bit >> 5;
  const int sh = (int)(bit & 31);
  const uint64_t a = ((uint64_t)in32[wi + 1] << 32) | in32[wi];
  uint64_t v = (a >> sh) | (sh ? (uint64_t)in32[wi + 2] << (64 - sh) : 0);
  uint64_t avail = nbytes * 8 > bit ? nbytes * 8 - bit : 0;
  int kk = avail < (uint64_t)k ? (int)avail : k;
  return kk ? v & (~0ull >> (64 - kk)) : 0;
}

// Kraft equality over 15-bit leaves, or a single one-bit code.
static __device__ __forceinline__ bool kraft_exact(uint32_t leaves, uint32_t gt1) {
  if (leaves == (1u << 14)) return gt1 == 0;
  return leaves == (1u << 15);
}

// Bits [bit, bit + 96) of the stream as (lo64, hi32), from four aligned
// 32-bit loads; bits at or past the stream end read 0 (the buffer is padded,
// so the loads stay inside it).
static __device__ __forceinline__ void load_bits96(const uint8_t* in, uint64_t nbytes,
                                                   uint64_t bit, uint64_t& x, uint32_t& xh) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint64_t wi = bit >> 5;
  const uint32_t w0 = in32[wi], w1 = in32[wi + 1], w2 = in32[wi + 2], w3 = in32[wi + 3];
  const int sh = (int)(bit & 31);
  const uint64_t a = ((uint64_t)w1 << 32) | w0, b = ((uint64_t)w3 << 32) | w2;
  x = sh ? (a >> sh) | (b << (64 - sh)) : a;
  xh = (uint32_t)(b >> sh);
  const uint64_t nbits = nbytes * 8;
  if (bit + 96 > nbits) {
    const uint64_t valid = nbits > bit ? nbits - bit : 0;
    if (valid < 64) {
      x &= valid ? (~0ull >> (64 - valid)) : 0;
      xh = 0;
    } else {
      xh &= valid > 64 ? (0xFFFFFFFFu >> (96 - valid)) : 0;
    }
  }
}

// Leaf count of 4 precode lengths (3 bits each) packed in 12 bits: the
// table of validate_precode (blockfinder_validation.rs:148-226).
static __device__ __forceinline__ uint32_t precode_leaves4(uint32_t v) {
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    uint32_t L = (v >> (3 * i)) & 7;
    s += L ? 1u << (7 - L) : 0u;
  }
  return s;
}

// Place of each code-length symbol in the header's order.
static __device__ __forceinline__ constexpr int precode_place(int sym) {
  constexpr int at[19] = {3, 17, 15, 13, 11, 9, 7, 5, 4, 6, 8, 10, 12, 14, 16, 18, 0, 1, 2};
  return at[sym];
}

// Rest of the dynamic-header predicate once the 13-bit filter and the
// precode leaf count have passed: Kraft-exact precode, code lengths decode,
// EOB present, Kraft-exact litlen and dist sets.  One thread per candidate,
// all state in registers (the canonical precode as 7 limits and the symbols
// in code order, 5 bits each): a candidate costs its serial chain of code
// lengths, so it must not wait for local memory on the way.
static __device__ __noinline__ bool dyn_candidate_full(const uint8_t* in, uint64_t nbytes,
                                                       uint64_t bit) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint64_t nbits = nbytes * 8;
  const uint32_t h = (uint32_t)peek_bits(in, nbytes, bit, 17);
  const int hl = 257 + (int)((h >> 3) & 31), total = hl + 1 + (int)((h >> 8) & 31);
  const int pc = (int)((h >> 13) & 15) + 4;
  const uint64_t pbits = peek_bits(in, nbytes, bit + 17, 3 * pc);
  // codes per length, eight bits each; length 0 is not counted
  uint64_t cnt = 0;
#pragma unroll
  for (int i = 0; i < 19; i++) cnt += 1ull << (8 * ((pbits >> (3 * i)) & 7));
  cnt &= ~0xFFull;
  uint32_t lim[8];  // left-aligned end of the codes of up to l bits
  uint64_t base = 0, next = 0;
  {
    uint32_t code = 0, off = 0, c = 0, leaves = 0, gt1 = 0;
#pragma unroll
    for (int l = 1; l < 8; l++) {
      code = (code + c) << 1;
      c = (uint32_t)(cnt >> (8 * l)) & 0xFF;
      lim[l] = (code + c) << (7 - l);
      base |= (uint64_t)((off - code) & 0xFF) << (8 * l);
      next |= (uint64_t)off << (8 * l);
      off += c;
      leaves += c << (15 - l);
      if (l > 1) gt1 += c;
    }
    if (!kraft_exact(leaves, gt1)) return false;
  }
  uint64_t s_lo = 0, s_hi = 0;  // symbols in code order: 12, then 7
#pragma unroll
  for (int sym = 0; sym < 19; sym++) {
    const uint32_t L = (uint32_t)(pbits >> (3 * precode_place(sym))) & 7;
    if (!L) continue;
    const uint32_t at = (uint32_t)(next >> (8 * L)) & 0xFF;
    next += 1ull << (8 * L);
    if (at < 12) s_lo |= (uint64_t)sym << (5 * at);
    else s_hi |= (uint64_t)sym << (5 * (at - 12));
  }
  // decode the litlen + dist code lengths, accumulating Kraft sums
  uint64_t pos = bit + 17 + 3 * pc;
  uint64_t wi = pos >> 5;
  uint64_t buf = in32[wi] >> (pos & 31);
  int have = 32 - (int)(pos & 31);
  wi++;
  uint32_t lit_leaves = 0, lit_gt1 = 0, dist_leaves = 0, dist_gt1 = 0;
  int i = 0;
  uint32_t prev = 0, eob_len = 0;
  while (i < total) {
    if (pos >= nbits) return false;
    if (have < 14) {
      buf |= (uint64_t)in32[wi++] << have;
      have += 32;
    }
    const uint32_t rev = __brev((uint32_t)buf) >> 25;  // MSB-first 7-bit code
    if (rev >= lim[7]) return false;
    uint32_t L = 1;
#pragma unroll
    for (int l = 1; l < 7; l++) L += rev >= lim[l] ? 1u : 0u;
    const uint32_t idx = ((rev >> (7 - L)) + (uint32_t)(base >> (8 * L))) & 0x1F;
    const uint32_t sym = (uint32_t)(idx < 12 ? s_lo >> (5 * idx) : s_hi >> (5 * (idx - 12))) & 31;
    // a repeat's bits: 2, 3 or 7
    const uint32_t xb = sym < 16 ? 0u : (sym == 16 ? 2u : (sym == 17 ? 3u : 7u));
    const uint32_t x = (uint32_t)(buf >> L) & ((1u << xb) - 1);
    if (sym == 16 && i == 0) return false;
    const uint32_t v = sym < 16 ? sym : (sym == 16 ? prev : 0u);
    const int rep = sym < 16 ? 1 : (int)x + (sym == 18 ? 11 : 3);
    buf >>= L + xb;
    have -= (int)(L + xb);
    pos += L + xb;
    if (i + rep > total || pos > nbits) return false;
    if (v) {
      const int n_lit = i < hl ? min(rep, hl - i) : 0;
      const int n_dist = rep - n_lit;
      lit_leaves += (uint32_t)n_lit << (15 - v);
      dist_leaves += (uint32_t)n_dist << (15 - v);
      if (v > 1) {
        lit_gt1 += n_lit;
        dist_gt1 += n_dist;
      }
      if (i <= 256 && 256 < i + rep) eob_len = v;
      // Kraft sums only grow: an over-subscribed set fails the final test
      if (lit_leaves > (1u << 15) || dist_leaves > (1u << 15)) return false;
    }
    prev = v;
    i += rep;
  }
  if (eob_len == 0) return false;
  return kraft_exact(lit_leaves, lit_gt1) && kraft_exact(dist_leaves, dist_gt1);
}

// The cheap part of the dynamic-header predicate at `bit`: the 13-bit header
// filter and the precode leaf count; dyn_candidate_fast adds
// dyn_candidate_full.
static __device__ __forceinline__ bool dyn_candidate_fast(const uint8_t* in, uint64_t nbytes,
                                                          uint64_t bit) {
  if (bit + 17 > nbytes * 8) return false;
  uint64_t x;
  uint32_t xh;
  load_bits96(in, nbytes, bit, x, xh);
  const uint32_t h = (uint32_t)x;
  if ((h & 1) || ((h >> 1) & 3) != 2 || ((h >> 3) & 31) > 29 || ((h >> 8) & 31) > 29) return false;
  const int pc = ((h >> 13) & 15) + 4;
  if (bit + 17 + 3 * pc > nbytes * 8) return false;
  // precode bits [17, 17 + 3*pc) of the 96-bit window
  uint64_t pb = (x >> 17) | ((uint64_t)xh << 47);
  pb &= (1ull << (3 * pc)) - 1;
  const uint32_t leaves =
      precode_leaves4((uint32_t)(pb & 0xFFF)) + precode_leaves4((uint32_t)((pb >> 12) & 0xFFF)) +
      precode_leaves4((uint32_t)((pb >> 24) & 0xFFF)) +
      precode_leaves4((uint32_t)((pb >> 36) & 0xFFF)) + precode_leaves4((uint32_t)(pb >> 48));
  return (leaves == 128 || leaves == 64) && dyn_candidate_full(in, nbytes, bit);
}

// The block after a true non-final stored block starts at byte `n` (its
// header's first bit is bit 0 of that byte): another stored block (LEN ==
// ~NLEN one byte on) or a dynamic block whose header passes the full
// predicate.  Not a rule of the reference's finder: it drops the false
// LEN/NLEN matches (about one per 64 KiB of random bytes) that would
// otherwise start speculative chunks inside stored data.  A true stored
// block followed by a fixed-Huffman block is given up as a start.  All but that
// predicate; kSuccHeader: it decides.
enum : int { kSuccNo = 0, kSuccYes = 1, kSuccHeader = 2 };
static __device__ __forceinline__ int stored_successor(const uint8_t* in, uint64_t nbytes, uint64_t n) {
  if (n >= nbytes) return kSuccNo;
  const uint32_t bt = (in[n] >> 1) & 3;
  if (bt == 0) {
    if (n + 5 > nbytes) return kSuccNo;
    const uint32_t sz = in[n + 1] | (in[n + 2] << 8) | ((uint32_t)in[n + 3] << 16) |
                        ((uint32_t)in[n + 4] << 24);
    return ((sz ^ (sz >> 16)) & 0xFFFF) == 0xFFFF ? kSuccYes : kSuccNo;
  }
  if (bt != 2) return kSuccNo;
  const uint64_t bit = n * 8;
  if (bit + 17 > nbytes * 8) return kSuccNo;
  const uint32_t h = (uint32_t)peek_bits(in, nbytes, bit, 13);
  if (((h >> 3) & 31) > 29 || ((h >> 8) & 31) > 29) return kSuccNo;
  return kSuccHeader;
}
// Stored candidate test at byte offset `off` (find_uncompressed_blocks):
// LEN == ~NLEN at the byte boundary, 3 zero header bits before it; the
// candidate spans [byte_bit - zero_run, byte_bit - 3].
static __device__ __forceinline__ bool stored_candidate(const uint8_t* in, uint64_t nbytes,
                                                        uint64_t off, uint64_t from, uint64_t to,
                                                        uint64_t hi_to, uint64_t& lo, uint64_t& hi) {
  uint32_t sz = in[off] | (in[off + 1] << 8) | ((uint32_t)in[off + 2] << 16) |
                ((uint32_t)in[off + 3] << 24);
  if (((sz ^ (sz >> 16)) & 0xFFFF) != 0xFFFF) return false;
  uint64_t byte_bit = off * 8;
  uint32_t pre = (uint32_t)peek_bits(in, nbytes, byte_bit - 10, 10);
  if (pre & (7u << 7)) return false;
  int tz = 3;
  for (int j = 4; j <= 10; j++) {
    if (pre & (1u << (10 - j))) break;
    tz = j;
  }
  lo = byte_bit - tz;
  hi = byte_bit - 3;
  uint32_t len = sz & 0xFFFF;
  return lo >= from && lo < to && hi < hi_to && len != 0 && off + 4 + len <= nbytes;
}

// Bits [p, p + 64) of the stream from three aligned 32-bit loads (the buffer
// is padded past the stream; bits past its end are not masked here).
static __device__ __forceinline__ uint64_t bits64_at(const uint32_t* in32, uint64_t p) {
  const uint64_t wi = p >> 5;
  const int sh = (int)(p & 31);
  const uint64_t a = ((uint64_t)in32[wi + 1] << 32) | in32[wi];
  return sh ? (a >> sh) | ((uint64_t)in32[wi + 2] << (64 - sh)) : a;
}

// Positions i < 32 (bit i of the result) where the 13-bit dynamic header
// filter passes, for the 64 stream bits X starting at the first of them:
// BFINAL = 0 (or either: any_final), BTYPE = 10, HLIT <= 29 (not bits 4..7 all set), HDIST <= 29
// (not bits 9..12 all set).  All 32 positions at once, bit-parallel.
static __device__ __forceinline__ uint32_t dyn_filter32(uint64_t X, bool any_final = false) {
  const uint64_t hlit_big = (X >> 4) & (X >> 5) & (X >> 6) & (X >> 7);
  const uint64_t hdist_big = (X >> 9) & (X >> 10) & (X >> 11) & (X >> 12);
  return (uint32_t)((any_final ? ~0ull : ~X) & ~(X >> 1) & (X >> 2) & ~hlit_big & ~hdist_big);
}

// Byte offsets k < 4 (bit k) among off .. off + 3 where LEN == ~NLEN, from
// the 7 bytes at off held in the low bits of B (bytes beyond are ignored).
static __device__ __forceinline__ uint32_t stored_filter4(uint64_t B) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t sz = (uint32_t)(B >> (8 * k));
    m |= (((sz ^ (sz >> 16)) & 0xFFFFu) == 0xFFFFu ? 1u : 0u) << k;
  }
  return m;
}

// First candidate in (bit_offset, seek_bit) order with bit_offset in
// [from, to) of the stream ending at byte `nbytes` (a stored candidate's
// seek bit must also be below hi_to); all 32 lanes call it together and get
// the same answer.  The range is walked in 1024-bit windows.  In each, every
// lane first screens 4 byte offsets for a stored block's LEN/NLEN pair, then
// 32 bit offsets with the 13-bit dynamic header filter, both bit-parallel,
// and runs the full tests only on the offsets that pass (about 1 in 9 bits);
// a ballot picks the lowest hit.  The first stored hit in byte order is the
// smallest stored candidate, so the dynamic scan only needs to reach it.
// Used by the inflate kernel's retry; the finder kernel screens ahead of it.
static __device__ bool warp_find_first(const uint8_t* __restrict__ in, uint64_t nbytes,
                                       uint64_t from, uint64_t to, uint64_t hi_to, int lane,
                                       uint64_t& out_lo, uint64_t& out_hi) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  if (to > nbytes * 8) to = nbytes * 8;
  if (hi_to > nbytes * 8) hi_to = nbytes * 8;
  bool have = false;
  uint64_t best_lo = 0, best_hi = 0;
  const uint64_t until = nbytes >= 5 ? min((hi_to + 7) / 8, nbytes - 4) : 0;
  uint64_t next_off = max((from + 3 + 7) / 8, (uint64_t)2);
  for (uint64_t w0 = from; w0 < to; w0 += 1024) {
    const uint64_t w1 = min(w0 + 1024, to);
    // stored offsets whose candidate may start below w1 (start >= off*8 - 10)
    const uint64_t off_end = min(until, (w1 + 10) / 8 + 1);
    while (!have && next_off < off_end) {
      const uint64_t ob = next_off + 4 * (uint64_t)lane;
      uint32_t m = 0;
      if (ob < off_end) {
        m = stored_filter4(bits64_at(in32, ob * 8));
        if (ob + 4 > off_end) m &= (1u << (off_end - ob)) - 1;
      }
      uint64_t lo = 0, hi = 0;
      bool hit = false;
      while (m) {
        const int k = __ffs(m) - 1;
        m &= m - 1;
        if (stored_candidate(in, nbytes, ob + k, from, to, hi_to, lo, hi)) {
          hit = true;
          break;
        }
      }
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, hit);
      if (b) {
        const int src = __ffs(b) - 1;
        best_lo = __shfl_sync(0xFFFFFFFFu, lo, src);
        best_hi = __shfl_sync(0xFFFFFFFFu, hi, src);
        have = true;
      }
      next_off = min(next_off + 128, off_end);
    }
    // dynamic candidates below the stored one (a tie at its bit_offset sorts first)
    const uint64_t lim = have ? min(w1, best_lo + 1) : w1;
    const uint64_t pl = w0 + 32 * (uint64_t)lane;
    uint32_t m = 0;
    if (pl < lim) {
      m = dyn_filter32(bits64_at(in32, pl));
      if (pl + 32 > lim) m &= (1u << (lim - pl)) - 1;
    }
    int hit = -1;
    while (m) {
      const int i = __ffs(m) - 1;
      m &= m - 1;
      if (dyn_candidate_fast(in, nbytes, pl + i)) {
        hit = i;
        break;
      }
    }
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, hit >= 0);
    if (b) {
      const int src = __ffs(b) - 1;
      const int i = __shfl_sync(0xFFFFFFFFu, hit, src);
      out_lo = out_hi = w0 + 32 * (uint64_t)src + (uint64_t)i;
      return true;
    }
    if (have && best_lo < w1) break;
  }
  out_lo = best_lo;
  out_hi = best_hi;
  return have;
}

// ---------------------------------------------------------------------------
// Sync starts in fixed-Huffman data (no counterpart in the reference, whose
// finder has no fixed-Huffman candidates: a fixed block has no header to
// test).  A walk decodes only positions with the fixed code of RFC 1951
// 3.2.6: a literal/length code, a length's extra bits, the 5-bit distance
// code and its extra bits; EOB must be followed by another fixed-block
// header.  Walks from a true symbol boundary never fail and all reach the
// same first boundary at or past the target; walks from a wrong bit fail
// (codes 286-287, distance codes 30-31, a non-fixed header) or fall into
// step with the true boundaries.  The search walks kSyncOffsets start bits
// and takes the end position most walks agree on (at least two; ties go to
// the lower position).  Whether that position really is a boundary is
// decided by the predecessor chunk, which hands over only on reaching it as
// a symbol start inside a non-final fixed block.
// ---------------------------------------------------------------------------
static __constant__ uint8_t f_len_extra[29] = {0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 2, 2, 2,
                                               2, 3, 3, 3, 3, 4, 4, 4, 4, 5, 5, 5, 5, 0};
static __constant__ uint8_t f_dist_extra[30] = {0, 0, 0, 0, 1, 1, 2, 2, 3, 3, 4, 4, 5, 5, 6,
                                                6, 7, 7, 8, 8, 9, 9, 10, 10, 11, 11, 12, 12, 13, 13};

// Walk entry of the 9 bits at a symbol start, fixed code: [4:0] bits of the
// code and a length's extra bits, [6:5] 0 literal, 1 length, 2 EOB, 3 invalid.
static __device__ __forceinline__ uint32_t fixed_entry(uint32_t x) {
  const uint32_t c7 = __brev(x & 127u) >> 25, c8 = __brev(x & 255u) >> 24;
  uint32_t sym, n;
  if (c7 <= 0x17) sym = 256 + c7, n = 7;
  else if (c8 <= 0xBF) sym = c8 - 0x30, n = 8;
  else if (c8 <= 0xC7) sym = 280 + (c8 - 0xC0), n = 8;
  else sym = 0, n = 9;  // 144 .. 255
  if (sym < 256) return n;
  if (sym == 256) return 2u << 5 | n;
  if (sym > 285) return 3u << 5;
  return 1u << 5 | (n + f_len_extra[sym - 257]);
}

// words a walk of `span` bits from a start inside `starts` bits stages
static __host__ __device__ constexpr uint32_t sync_words(uint64_t starts, uint64_t span) {
  return (uint32_t)((starts + span + 96 + 64) / 32) + 2;
}


// ---------------------------------------------------------------------------
// Expected output bytes per compressed byte of the dynamic block whose header
// starts at `bit` (a candidate the finder accepted), from its code lengths
// alone: a code of length L stands for a symbol of probability 2^-L.
// Literals give one byte, a length symbol its mean length; a symbol costs its
// code, its extra bits and, for a length, the mean distance code and extra
// bits.  Used to cut high-ratio partitions finer (no reference counterpart).
// ---------------------------------------------------------------------------
static __constant__ uint16_t f_len_base[29] = {3,  4,  5,  6,  7,  8,  9,  10, 11,  13,
                                               15, 17, 19, 23, 27, 31, 35, 43, 51,  59,
                                               67, 83, 99, 115, 131, 163, 195, 227, 258};

static __device__ __noinline__ float dyn_header_ratio(const uint8_t* in, uint64_t nbytes,
                                                      uint64_t bit) {
  const uint32_t h = (uint32_t)peek_bits(in, nbytes, bit, 17);
  const int hl = 257 + ((h >> 3) & 31), hd = 1 + ((h >> 8) & 31), pc = ((h >> 13) & 15) + 4;
  const uint64_t pbits = peek_bits(in, nbytes, bit + 17, 3 * pc);
  uint8_t cl[19];
  for (int i = 0; i < 19; i++) cl[i] = 0;
  for (int i = 0; i < pc; i++) cl[f_cl_order[i]] = (uint8_t)((pbits >> (3 * i)) & 7);
  uint16_t cnt[8], first[8], offs[8];
  uint8_t sorted[19];
  for (int L = 0; L < 8; L++) cnt[L] = 0;
  for (int s = 0; s < 19; s++) cnt[cl[s]]++;
  cnt[0] = 0;
  {
    uint32_t code = 0, off = 0;
    for (int L = 1; L < 8; L++) {
      if (L > 1) code = (code + cnt[L - 1]) << 1;
      first[L] = (uint16_t)code;
      offs[L] = (uint16_t)off;
      off += cnt[L];
    }
    uint16_t nx[8];
    for (int L = 0; L < 8; L++) nx[L] = offs[L];
    for (int s = 0; s < 19; s++)
      if (cl[s]) sorted[nx[cl[s]]++] = (uint8_t)s;
  }
  float out = 0.f, bits = 0.f, len_p = 0.f, dist_bits = 0.f, dist_p = 0.f;
  uint64_t pos = bit + 17 + 3 * pc;
  const int total = hl + hd;
  uint32_t prev = 0;
  for (int i = 0; i < total;) {
    const uint32_t rev = __brev((uint32_t)peek_bits(in, nbytes, pos, 14)) >> 25;
    int sym = -1;
    for (int L = 1; L < 8; L++) {
      const uint32_t idx = (rev >> (7 - L)) - first[L];
      if (idx < cnt[L]) {
        sym = sorted[offs[L] + idx];
        pos += L;
        break;
      }
    }
    if (sym < 0) return 0.f;
    uint32_t v = (uint32_t)sym;
    int rep = 1;
    if (sym == 16) {
      v = prev;
      rep = 3 + (int)peek_bits(in, nbytes, pos, 2);
      pos += 2;
    } else if (sym == 17) {
      v = 0;
      rep = 3 + (int)peek_bits(in, nbytes, pos, 3);
      pos += 3;
    } else if (sym == 18) {
      v = 0;
      rep = 11 + (int)peek_bits(in, nbytes, pos, 7);
      pos += 7;
    }
    if (v) {
      const float p = __int_as_float((127 - (int)v) << 23);  // 2^-v
      for (int k = i; k < i + rep && k < total; k++) {
        if (k < 256) {
          out += p;
          bits += p * (float)v;
        } else if (k >= 257 && k < hl && k < 286) {
          const int li = k - 257;
          len_p += p;
          out += p * ((float)f_len_base[li] + 0.5f * (float)((1u << f_len_extra[li]) - 1));
          bits += p * (float)(v + f_len_extra[li]);
        } else if (k >= hl) {
          const int di = k - hl;
          if (di < 30) {
            dist_p += p;
            dist_bits += p * (float)(v + f_dist_extra[di]);
          }
        }
      }
    }
    prev = v;
    i += rep;
  }
  if (dist_p > 0.f) bits += len_p * dist_bits / dist_p;
  return bits > 0.f ? 8.f * out / bits : 0.f;
}

}  // namespace gzgpu

