// block_cta.cuh -- one CTA decodes one chunk (page history).
//
// Block body.  A Huffman-coded block is decoded in rounds of up to
// NT (the CTA's threads, 256 or 1,024) bit ranges of `r` bits each, one range per
// thread:
//   1. every thread walks its range from a guessed start (its first bit),
//      following symbol lengths only.  Prefix codes resynchronise: a walk that
//      starts off a symbol boundary falls into step with the true one, so most
//      ranges end at the right bit although they started at a wrong one.
//   2. each range is walked again from where the range before it ended, and
//      again while that end moves, until no start changes (or all ranges up
//      to one that met the end of the block agree).  By induction from the
//      first range, whose start is exact, the joined ranges are the serial
//      decode.  Each pass confirms at least one more range.  A walk leaves
//      the first boundary past the half of its range, and the lookups from
//      there to its end; a later walk that meets one of them is done.
//   3. a block scan of the ranges' lookup counts gives each its place in the
//      round's token list (a literal: one slot; a match: length, then
//      distance), written by one decode of each range.
//   4. the tokens are expanded in windows of kWin output positions (see
//      expand_tokens), which leave as coalesced stores to the pages.
// Threads leave the data-dependent loops at different times; every barrier of
// the CTA joins each warp's lanes first (barrier.cuh).
// What bounds a block is its serial chain of code lookups; the ranges cut
// that chain into up to NT pieces.  Ranges of 512 bits end in step after a
// wrong start for 98 % of text, 88 % of byte runs and 59 % of noisy ramps
// (codes nearly all of one length), measured on zlib level 6 streams.
// Inflate kernel, before (one warp per chunk, steps of 64 bits decoded by the
// whole warp) and now: 64 MiB text 6.9 -> 0.56 ms, 12 MiB ramps 4.6 -> 0.45,
// 64 MiB byte runs 22 -> 0.45, 16 MiB of fixed codes 7.8 -> 0.25, a 4 KiB
// stream 0.195 -> 0.044.  Where the cycles go (text; ramps): expansion 55 %;
// 23 %, joining the ranges 12; 49, tokens 9; 7, guessed walks 8; 7, tables and
// headers 13; 12.
#pragma once
#include <cstdint>

#include "barrier.cuh"
#include "common.cuh"
#include "huffman.cuh"
#include "inflate.cuh"

namespace gzgpu {

constexpr uint32_t kRangeMax = 640;   // bits per thread and round, at most
// and at least: shorter ranges fall into step in too few of them (passes over
// 3.4 times the ranges of text at 256 bits, 7 at 128), and must be longer than
// a symbol (48)
constexpr uint32_t kRangeMin = 256;
constexpr uint32_t kWinPer = 8;         // output positions expanded at a time, per thread
constexpr uint32_t kTokPer = 4;       // token slots per thread and batch
constexpr uint32_t kCtaDistBits = 9;  // distance LUT index bits
constexpr uint32_t kSegs = 2;           // a range is walked in halves
// a block header's code lengths: bits (316 codes of 7 bits, or fewer symbols)
// and symbols at most
constexpr uint32_t kHdrBits = 2240;
constexpr uint32_t kHdrSyms = 320;
constexpr uint32_t kNone = 0xFFFFFFFFu;

// Table entry: [4:0] bits of the code and its extra bits, bit 5 = length code,
// [23:8] token value without the extra bits, [30:27] code length; bit 31 =
// not a literal, length or distance: end of block, or, by value, invalid, or
// not in the LUT ([4:0] = 0; bit 5 = the distance LUT's).  The shift amounts sit where the shifts read them, so the
// chain from one lookup to the next is mask, load, shift.
enum : uint32_t { kEntLen = 0x20, kEntStop = 0x80000000u };
enum : uint32_t { kStopEob = 0, kStopBad = 1, kStopLong = 2 };
constexpr uint32_t kTokMatch = 0x8000u;  // a match's first slot: flag and length

__device__ __forceinline__ uint32_t tok_lit_entry(uint32_t sym, uint32_t L) {
  if (sym < 256) return L << 27 | sym << 8 | L;
  if (sym == 256) return kEntStop | L << 27 | kStopEob << 8;
  if (sym <= 285) {
    const uint32_t k = sym - 257;
    return L << 27 | (kTokMatch + c_len_base[k]) << 8 | kEntLen | (L + c_len_extra[k]);
  }
  return kEntStop | kStopBad << 8;
}
__device__ __forceinline__ uint32_t tok_dist_entry(uint32_t sym, uint32_t L) {
  if (sym < 30) return L << 27 | (uint32_t)(c_dist_base[sym] - 1) << 8 | (L + c_dist_extra[sym]);
  return kEntStop | kEntLen | kStopBad << 8;
}

// the chunk's state, written by thread 0 (or warp 0) and read by all after a barrier
struct CtaCtl {
  uint64_t pos, o;          // next input bit, entries written
  uint64_t stop_lo, abort_bit, slack, limit_words, trunc_words, in_end, table_bit;
  uint64_t hdr_pos;         // first bit after a dynamic header's precode
  uint64_t blk_hdr;         // header bit of the block being decoded (0 = unknown)
  uint64_t marker_end, sync_target, passed_bit;
  uint64_t cand_lo, cand_hi;
  uint64_t t0;
  uint32_t next, flags, cid, gen;
  uint32_t bfinal, btype, n_blocks, extends, stored_len;
  int32_t act, status;
  uint32_t nlen, ndist, final_block, synced, passed, resume, in_sync_block;
  uint32_t spec, again;     // speculative start; try the next candidate
  uint32_t fixed_tables;    // the tables in place are the fixed code's
  // move pos past the header; its length after hdr_pos; where the symbol that
  // ends its reading, the last or the first wrong one, begins after it
  uint32_t hdr_move, hdr_end, hdr_last;
  uint32_t build_ok[2];
  uint32_t page_cur, page_prev, page_seq, n_pages;
  uint32_t round_slots, round_lanes, round_kind, round_pos;
  int32_t carry_ms;         // match reaching into the next window: start (relative to it)
  uint32_t carry_len, carry_dist;
  uint32_t mark_max;
};

// A code beside its LUT: codes are canonical, so the length of the code at the
// head of a 15-bit window (first bit = MSB) is the number of lengths l with
// window >= lim[l], plus one, and its place among the codes sorted by length
// and symbol is (window >> (15 - length)) + base[length].
struct CodeIndex {
  uint32_t lim[16], base[16];
  uint16_t count[16], offs[16];
};

template <int LB, int NT>
struct alignas(16) CtaSmem {
  static constexpr uint32_t kWin = NT * kWinPer;
  static constexpr uint32_t kTokCap = NT == 256 ? 18432 : 40960;  // token slots per round
  // literal/length LUT, then the distance LUT (at a power of two, so that its
  // offset joins an index by OR)
  uint32_t lut[(1 << LB) + (1 << kCtaDistBits)];
  union {
    uint16_t tok[kTokCap + 8];
    uint16_t hop[4][kHdrBits];  // block header: position 1, 2, 4 and 8 symbols on
    uint16_t list[NT];          // join: the ranges to walk again
  };
  union {
    struct {  // block header
      uint8_t lens[320];        // literal/length codes at 0, distance codes at 288
      uint8_t pre_lens[32];
      uint32_t pre_lut[128];
      uint16_t group[kHdrSyms / 8];  // position of every eighth symbol
      uint8_t val[kHdrSyms];         // a symbol's length, 0xFF: that of the one before
    };
    struct {          // expansion
      // two windows, by turns
      alignas(16) uint32_t stage[2][kWin];
      uint32_t bm[2][kWin / 32];  // match starts
    };
  };
  uint32_t lit_ent[288], dist_ent[32];  // entries in canonical order
  CodeIndex lit, dist;
  // the round's ranges: where each starts and ends, [15:0] its lookups (a
  // literal is one, a match two), [17:16] what ended it early and at which bit
  uint32_t start[NT], end[NT], info[NT], term_pos[NT];
  uint32_t need[NT / 32], term[NT / 32];
  // per part of each range but the last: [9:0] first boundary at or past
  // its end, relative to the range's first bit, [31:10] lookups from there
  uint32_t cp[kSegs - 1][NT];
  uint32_t scan[2][NT / 32];
  CtaCtl c;
};

// exclusive prefix sum of a over the CTA, total in ta.  One barrier; `par`
// alternates between calls (0, 1, 0, ...).
template <int LB, int NT>
__device__ __forceinline__ uint32_t cta_scan(CtaSmem<LB, NT>* S, uint32_t par, uint32_t a, uint32_t& ta) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = a;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if (lane >= d) x += u;
  }
  if (lane == 31) S->scan[par][warp] = x;
  cta_sync();
  uint32_t pa = 0;
  ta = 0;
  if constexpr (NT <= 256) {
#pragma unroll
    for (int w = 0; w < NT / 32; w++) {
      const uint32_t u = S->scan[par][w];
      if (w < warp) pa += u;
      ta += u;
    }
  } else {  // the warps' totals by the same scan
    const uint32_t own = lane < NT / 32 ? S->scan[par][lane] : 0u;
    uint32_t y = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, y, d);
      if (lane >= d) y += u;
    }
    pa = __shfl_sync(0xFFFFFFFFu, y - own, warp);
    ta = __shfl_sync(0xFFFFFFFFu, y, 31);
  }
  return pa + x - a;
}

// The entry of a code longer than the LUT's bits (9 for distances, 10 or more
// for literals and lengths), or kStopBad.  Inlined where it is used: a call in
// the walks' loops, taken or not, cost 30 cycles an iteration.
template <int LB, int NT>
__device__ __forceinline__ uint32_t long_entry(const CtaSmem<LB, NT>* S, uint32_t x, bool dist) {
  static_assert(LB >= 10 && kCtaDistBits == 9, "codes looked up here have 10 bits at least");
  const CodeIndex& I = dist ? S->dist : S->lit;
  const uint32_t rev = __brev(x) >> 17;  // 15 code bits, first bit = MSB
  uint32_t L = 10;
#pragma unroll
  for (int l = 10; l <= 15; l++) L += rev >= I.lim[l] ? 1u : 0u;
  if (L > 15) return kEntStop | (dist ? kEntLen : 0u) | kStopBad << 8;
  const uint32_t i = (rev >> (15 - L)) + I.base[L];
  return dist ? S->dist_ent[i] : S->lit_ent[i];
}

// One thread's bits: the next `q - p + 30` stream bits at bit 2 of hi:lo
// (indexes into the LUT are byte offsets), the word after them in w.  No
// branches: a divergent one costs about as much as a lookup.
struct RangeBits {
  const uint32_t* next;  // word after w
  uint32_t lo, hi, w;
  uint32_t p, q;  // position; refill when p >= q, which leaves 30 bits at least

  __device__ __forceinline__ void refill_if_due() {
    // 2 + the bits left (2 .. 32) is where the next word goes
    asm("{\n\t"
        ".reg .pred due;\n\t"
        ".reg .u32 s, a, b;\n\t"
        "setp.ge.u32 due, %4, %3;\n\t"
        "sub.u32 s, %3, %4;\n\t"
        "add.u32 s, s, 32;\n\t"
        "shf.l.clamp.b32 a, 0, %2, s;\n\t"
        "shf.l.clamp.b32 b, %2, 0, s;\n\t"
        "@due or.b32 %0, %0, a;\n\t"
        "@due or.b32 %1, %1, b;\n\t"
        "@due add.u32 %3, %3, 32;\n\t"
        "@due ld.global.u32 %2, [%5];\n\t"
        "@due add.u64 %5, %5, 4;\n\t"
        "}"
        : "+r"(lo), "+r"(hi), "+r"(w), "+r"(q), "+r"(p), "+l"(next));
  }
  // base: the word of position 0
  __device__ __forceinline__ void seek(const uint32_t* base, uint32_t pos) {
    const uint32_t* a = base + (pos >> 5);
    const uint32_t x = a[0] >> (pos & 31);
    w = a[1];
    next = a + 2;
    lo = x << 2;
    hi = x >> 30;
    p = pos;
    q = (pos & ~31u) + 2;  // 32 - (pos & 31) bits in place
    refill_if_due();
  }
  __device__ __forceinline__ void shift(uint32_t ent) {  // by ent[4:0] bits
    lo = __funnelshift_r(lo, hi, ent);
    hi = __funnelshift_r(hi, 0, ent);
    p += ent & 31;
  }
};

// what ended a range's walk before its end
enum : uint32_t { kTermNone = 0, kTermEob = 1, kTermBad = 2 };
constexpr uint32_t kNoCp = 0x3FFu;  // a part without a recorded boundary

enum : uint32_t { kInfoTerm = 1u << 16, kInfoOn = 1u << 18 };  // On: went on past a stop, starts nowhere

// The two tables as one: the byte offset of the current one (0: literals and
// lengths) and its index mask.  A stop entry keeps the table it came from.
template <int LB>
struct TableAt {
  uint32_t off = 0, mask = ((1u << LB) - 1) << 2;
  __device__ __forceinline__ uint32_t look(const char* lut, const RangeBits& b) const {
    return *reinterpret_cast<const uint32_t*>(lut + ((b.lo & mask) | off));
  }
  __device__ __forceinline__ void after(uint32_t ent) {
    off = ent & kEntLen ? 4u << LB : 0u;
    mask = off ? ((1u << kCtaDistBits) - 1) << 2 : ((1u << LB) - 1) << 2;
  }
};

// Walk range `id`, [first, first + len) cut at e, from its start on (S->start),
// positions relative to `base`.  A lookup is a literal or a length code, or the distance
// code of the length just read, so threads at literals and threads inside
// matches run the same instructions.  Four lookups per loop: a lookup that is
// not due (past the end, or too few bits before the next refill) takes nothing,
// which is cheaper than branching around it (warp alone: 143 cycles a lookup
// one by one, 100 so; 24 warps: 216 and 165).  guess: the start may be no
// symbol boundary; go on past a stop (from the next bit) to find a likely end
// for the range.  Otherwise a stop ends the walk.  again: an earlier walk of
// this round left its boundaries, and meeting one ends this walk: from there
// on they agree.
template <int LB, int NT>
__device__ __forceinline__ void walk_range(CtaSmem<LB, NT>* S, const uint32_t* base, uint32_t first,
                                           uint32_t len, uint32_t e, uint32_t id, bool guess,
                                           bool again) {
  const char* lut = reinterpret_cast<const char*>(S->lut);
  RangeBits b;
  b.seek(base, S->start[id]);
  TableAt<LB> t;
  uint32_t slots = 0, valid_from = 0, seg = 0;
  uint32_t term = kTermNone;
  bool met = false, on = false;
  for (;; seg++) {
    uint32_t es = seg == kSegs - 1 ? e : min(e, first + (seg + 1) * (len / kSegs));
    if (b.p < es) do {
      uint32_t stop = 0;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const bool due = b.p < (t.off ? kNone : es) && (u % 2 == 0 || b.p < b.q);
        const uint32_t ent = due ? t.look(lut, b) : 0u;
        b.shift(ent);
        slots += (int32_t)ent > 0 ? 1u : 0u;
        if (due) t.after(ent);
        stop |= ent;
        if (u % 2) b.refill_if_due();
      }
      if (__builtin_expect((int32_t)stop < 0, 0)) {
        // at p: a code beyond the LUT, or a stop
        const bool dist = t.off != 0;
        uint32_t ent = t.look(lut, b);
        if (((ent >> 8) & 3) == kStopLong) ent = long_entry<LB, NT>(S, b.lo >> 2, dist);
        if ((int32_t)ent >= 0) {
          slots++;
        } else if (guess) {
          on = true;
          valid_from = seg;  // boundaries before the stop lead to it
          slots++;
          ent = 1;           // one bit on
        } else {
          const bool eob = ((ent >> 8) & 3) == kStopEob;
          term = eob ? kTermEob : kTermBad;
          S->term_pos[id] = b.p + (eob ? (ent >> 27) & 15 : 0u);
          ent = 0;
          es = 0;  // ends the walk
        }
        b.shift(ent);
        b.refill_if_due();
        t.after(ent);
      }
    } while (b.p < (t.off ? kNone : es));
    if (term || seg == kSegs - 1) break;
    const uint32_t at = b.p - first;
    if (again) {
      const uint32_t old = S->cp[seg][id];
      if ((old & 0x3FFu) == at) {
        slots += old >> 10;
        met = true;
        break;
      }
    }
    S->cp[seg][id] = at | slots << 10;
  }
  // seg parts were passed; their lookups become those left to the end
  for (uint32_t k = 0; k < kSegs - 1; k++) {
    if (term || (guess && k < valid_from)) S->cp[k][id] = kNoCp;
    else if (k < seg) S->cp[k][id] = (S->cp[k][id] & 0x3FFu) | (slots - (S->cp[k][id] >> 10)) << 10;
  }
  S->info[id] = slots | term * kInfoTerm | (on ? kInfoOn : 0u);
  if (!term && !met) S->end[id] = b.p;
}

// The tokens of the n lookups from start on to tok.
template <int LB, int NT>
__device__ __forceinline__ void write_tokens(const CtaSmem<LB, NT>* S, const uint32_t* base,
                                             uint32_t start, uint32_t n, uint16_t* tok) {
  const char* lut = reinterpret_cast<const char*>(S->lut);
  RangeBits b;
  b.seek(base, start);
  TableAt<LB> t;
  uint16_t* const end = tok + n;
  while (tok < end) {
    uint32_t stop = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const bool due = tok < end && (u % 2 == 0 || b.p < b.q);
      const uint32_t ent = due ? t.look(lut, b) : 0u;
      if ((int32_t)ent > 0) {
        // value + extra bits: the code's bits cut off the front of what it takes
        const uint32_t x = (b.lo >> 2) & ~(0xFFFFFFFFu << (ent & 31));
        *tok++ = (uint16_t)((ent >> 8) + (x >> (ent >> 27)));
      }
      b.shift(ent);
      if (due) t.after(ent);
      stop |= ent;
      if (u % 2) b.refill_if_due();
    }
    if (__builtin_expect((int32_t)stop < 0, 0)) {
      const uint32_t ent = long_entry<LB, NT>(S, b.lo >> 2, t.off != 0);
      const uint32_t x = (b.lo >> 2) & ~(0xFFFFFFFFu << (ent & 31));
      *tok++ = (uint16_t)((ent >> 8) + (x >> (ent >> 27)));
      b.shift(ent);
      b.refill_if_due();
      t.after(ent);
    }
  }
}

// A code's index by one warp: counts, first codes, limits, and the symbols'
// entries in canonical order.  lens[0..n) in shared memory, n <= 320.
// Acceptance follows zlib (canon_build).
template <typename EntryFn>
__device__ __noinline__ bool index_code(const uint8_t* lens, int n, CodeIndex* I, uint32_t* ent,
                                        int lane, EntryFn entry) {
  if (lane < 16) I->count[lane] = 0;
  __syncwarp();
  // rank of each symbol among those of its length, in symbol order
  uint32_t rank[10], len[10];
#pragma unroll
  for (int g = 0; g < 10; g++) {
    const int s = 32 * g + lane;
    len[g] = s < n ? lens[s] : 0;
    rank[g] = 0;
    if (32 * g >= n) continue;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, len[g]);
    const uint32_t before = I->count[len[g]];
    rank[g] = before + __popc(peers & ((1u << lane) - 1));
    __syncwarp();
    if (len[g] && (__ffs(peers) - 1) == lane) I->count[len[g]] = (uint16_t)(before + __popc(peers));
    __syncwarp();
  }
  // lane L: first code, offset and limit of length L; Kraft sum in units of 2^-15
  const uint32_t cnt = lane >= 1 && lane <= 15 ? I->count[lane] : 0;
  uint32_t first = 0, offs = 0, kraft = 0, maxl = 0;
#pragma unroll
  for (int l = 1; l <= 15; l++) {
    const uint32_t c = __shfl_sync(0xFFFFFFFFu, cnt, l);
    if (l < lane) {
      first += c << ((lane - l) & 31);
      offs += c;
    }
    kraft += c << (15 - l);
    if (c) maxl = l;
  }
  if (lane >= 1 && lane <= 15) {
    I->lim[lane] = (first + cnt) << (15 - lane);
    I->base[lane] = offs - first;
    I->offs[lane] = (uint16_t)offs;
  }
  const bool ok = kraft <= 1u << 15 && (kraft == 1u << 15 || maxl <= 1);
  __syncwarp();
  if (!ok) return false;
#pragma unroll
  for (int g = 0; g < 10; g++)
    if (len[g]) ent[I->offs[len[g]] + rank[g]] = entry(32u * g + lane, len[g]);
  __syncwarp();
  return true;
}

// LUT entry i: the entry of the code at the head of i's low TB bits
template <int TB>
__device__ __forceinline__ uint32_t lut_value(uint32_t i, const uint32_t* lim, const CodeIndex* I,
                                              const uint32_t* ent, uint32_t longer) {
  const uint32_t rev = __brev(i) >> 17;
  uint32_t L = 1;
#pragma unroll
  for (int l = 1; l <= TB; l++) L += rev >= lim[l] ? 1u : 0u;
  if (L > TB) return longer;
  return ent[(rev >> (15 - L)) + I->base[L]];
}

// The code lengths of a dynamic block's header into S->lens (whole CTA): the
// precode's lengths are in S->pre_lens and indexed (S->lit), S->c.pos is the
// first bit after them.  A symbol's place depends on all before it, 200 and
// more of them one after another (150 cycles each when a warp read them so, a
// fifth of the decode of a 16 KB block).  Here every bit position is decoded as
// if a symbol started there; two, four and eight symbols on follow by doubling,
// so one thread takes eight symbols a step, and the symbols on that chain are
// then expanded in parallel.  Returns kOk or an error status; S->c.pos moves
// past the header.
template <int LB, int NT>
__device__ __forceinline__ int32_t cta_read_lens(const uint8_t* __restrict__ in, CtaSmem<LB, NT>* S,
                                                 bool move) {
  const uint32_t tid = threadIdx.x;
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint64_t pos = S->c.hdr_pos, w0 = pos >> 5, trunc = S->c.trunc_words;
  const uint32_t nlen = S->c.nlen, total = nlen + S->c.ndist;
  if (tid < 128) {
    const uint32_t rev = __brev(tid) >> 17;
    uint32_t L = 1;
#pragma unroll
    for (int l = 1; l <= 7; l++) L += rev >= S->lit.lim[l] ? 1u : 0u;
    S->pre_lut[tid] = L > 7 ? 0u : S->lit_ent[(rev >> (15 - L)) + S->lit.base[L]];
  }
  for (uint32_t i = tid; i < 320; i += NT) S->lens[i] = 0;
  cta_sync();
  // [4:0] symbol, [12:8] bits taken (0: no such code), [23:16] lengths covered
  auto at = [&](uint32_t i) {
    const uint32_t p = (uint32_t)(pos & 31) + i, j = p >> 5;
    const uint32_t a = w0 + j < trunc ? in32[w0 + j] : 0u, b = w0 + j + 1 < trunc ? in32[w0 + j + 1] : 0u;
    const uint32_t x = __funnelshift_r(a, b, p & 31);
    const uint32_t e = S->pre_lut[x & 127], L = e & 15, sym = e >> 16;
    if (L == 0) return 0u;
    const uint32_t xb = sym < 16 ? 0u : (sym == 16 ? 2u : (sym == 17 ? 3u : 7u));
    const uint32_t rep = sym < 16 ? 1u : ((x >> L) & ((1u << xb) - 1)) + (sym == 18 ? 11u : 3u);
    return sym | (L + xb) << 8 | rep << 16;
  };
  for (uint32_t i = tid; i < kHdrBits; i += NT) {
    const uint32_t n = (at(i) >> 8) & 31;
    S->hop[0][i] = n && i + n < kHdrBits ? (uint16_t)(i + n) : (uint16_t)0xFFFF;
  }
  cta_sync();
  for (int k = 0; k < 3; k++) {
    for (uint32_t i = tid; i < kHdrBits; i += NT) {
      const uint32_t h = S->hop[k][i];
      S->hop[k + 1][i] = h == 0xFFFF ? (uint16_t)0xFFFF : S->hop[k][h];
    }
    cta_sync();
  }
  if (tid == 0) {
    uint32_t p = 0;
    for (uint32_t g = 0; g < kHdrSyms / 8; g++) {
      S->group[g] = (uint16_t)p;
      if (p != 0xFFFF) p = S->hop[3][p];
    }
  }
  cta_sync();
  // symbols 2 tid and 2 tid + 1
  uint32_t e[2] = {0, 0}, p[2] = {0xFFFF, 0xFFFF};
  if (tid < kHdrSyms / 2) {
    p[0] = S->group[tid >> 2];
    if ((tid & 1) && p[0] != 0xFFFF) p[0] = S->hop[1][p[0]];
    if ((tid & 2) && p[0] != 0xFFFF) p[0] = S->hop[2][p[0]];
    if (p[0] != 0xFFFF) {
      e[0] = at(p[0]);
      p[1] = S->hop[0][p[0]];
      if (p[1] != 0xFFFF) e[1] = at(p[1]);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t sym = e[k] & 31;
      S->val[2 * tid + k] = sym < 16 ? (uint8_t)sym : (sym == 16 ? (uint8_t)0xFF : (uint8_t)0);
    }
  }
  uint32_t sum;
  uint32_t o = cta_scan(S, 0, (e[0] >> 16) + (e[1] >> 16), sum);
  if (tid == 0) S->c.hdr_end = S->c.hdr_last = kNone;
  cta_sync();
  uint32_t wrong = kNone;  // where this thread's first wrong symbol begins
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const uint32_t n = e[k] >> 16;
    if (tid < kHdrSyms / 2 && o < total) {
      uint32_t s = 2 * tid + k;
      if (!n || o + n > total || (s == 0 && (e[k] & 31) == 16)) {
        wrong = min(wrong, p[k]);
      } else {
        if (o + n == total) {
          S->c.hdr_end = p[k] + ((e[k] >> 8) & 31);
          S->c.hdr_last = p[k];
        }
        while (s && S->val[s] == 0xFF) s--;
        const uint8_t v = S->val[s];
        if (v)
          for (uint32_t j = o; j < o + n; j++) S->lens[j < nlen ? j : 288 + j - nlen] = v;
      }
    }
    o += n;
  }
  bool bad = cta_sync_or(wrong != kNone);
  if (bad) {
    if (wrong != kNone) atomicMin(&S->c.hdr_last, wrong);
    cta_sync();
  }
  bad = bad || S->c.hdr_end == kNone || S->lens[256] == 0;
  // Past the readable input (a serial reader ran 96 bits ahead of the symbol it
  // stopped at): cut off, or over the abort bit, whatever the lengths say.
  const uint64_t end = pos + S->c.hdr_end, ahead = pos + S->c.hdr_last + 96;
  cta_sync();
  if (ahead >= S->c.limit_words * 32) return ahead >= trunc * 32 ? kTruncated : kOvershoot;
  if (bad) return kBadDeflate;
  if (tid == 0 && move) S->c.pos = end;
  cta_sync();
  return kOk;
}

// Both code tables from S->lens (whole CTA).  Warp 0 sorts the
// literal/length code, warp 1 the distance code, all threads fill the LUT.
// Distance lengths sit at lens + 288.
template <int LB, int NT>
__device__ __forceinline__ bool cta_build_tables(CtaSmem<LB, NT>* S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < 2) {
    bool ok;
    if (warp == 0)
      ok = index_code(S->lens, (int)S->c.nlen, &S->lit, S->lit_ent, lane, tok_lit_entry);
    else
      ok = index_code(S->lens + 288, (int)S->c.ndist, &S->dist, S->dist_ent, lane, tok_dist_entry);
    if (lane == 0) S->c.build_ok[warp] = ok;
  }
  cta_sync();
  if (!S->c.build_ok[0] || !S->c.build_ok[1]) return false;
  uint32_t lim[LB + 1];
#pragma unroll
  for (int l = 1; l <= LB; l++) lim[l] = S->lit.lim[l];
  for (uint32_t i = threadIdx.x; i < (1u << LB); i += NT)
    S->lut[i] = lut_value<LB>(i, lim, &S->lit, S->lit_ent, kEntStop | kStopLong << 8);
#pragma unroll
  for (int l = 1; l <= (int)kCtaDistBits; l++) lim[l] = S->dist.lim[l];
  for (uint32_t i = threadIdx.x; i < (1u << kCtaDistBits); i += NT)
    S->lut[(1u << LB) + i] = lut_value<(int)kCtaDistBits>(i, lim, &S->dist, S->dist_ent,
                                                          kEntStop | kEntLen | kStopLong << 8);
  cta_sync();
  return true;
}

// Make the page of the window at chunk position w0 current (thread 0
// allocates, then a barrier).  Windows are visited in order and never cross a
// page.  False when the pool is exhausted.
template <int LB, int NT>
__device__ __forceinline__ bool cta_page(CtaSmem<LB, NT>* S, const PagePool& pool, uint64_t w0) {
  const uint32_t s = (uint32_t)(w0 >> 16);
  if (S->c.page_cur != kNoPage && S->c.page_seq == s) return true;
  cta_sync();
  if (threadIdx.x == 0) {
    uint32_t p = atomicAdd(pool.next, 1u);
    if (p < pool.cap) {
      pool.owner[p] = S->c.cid;
      pool.seq[p] = (S->c.gen << kGenShift) | s;
    } else {
      p = kNoPage;
    }
    S->c.page_prev = S->c.page_cur;
    S->c.page_cur = p;
    S->c.page_seq = s;
    S->c.n_pages++;
  }
  cta_sync();
  return S->c.page_cur != kNoPage;
}

// Expand a round's tokens (slots [0, n)) after the chunk's entry position
// S->c.o, and move that on (thread 0, before a barrier).  Output goes in windows of kWin positions
// aligned to kWin, so a window lies in one page.  Batches of kTokPer slots a
// thread get their positions from a block scan; literals and match records go
// to the window's stage (a match's record at its first position, a bit in
// bm).  Then every thread takes kWinPer positions in a row, finds the match
// that reaches into them and those that start in them, and gives each covered
// position its source: the history in the pages (or the marker / zero before
// the chunk), or a position of this window, followed by pointer jumping
// through the stage.  Neighbours mostly share a match, so a match is looked at
// once per thread, its sources are loaded from one address, and the window
// leaves in 16-byte stores; a window without matches goes out as it is.  The
// stage has two turns, so a window needs three barriers: its tokens are placed
// (which also makes the window before it readable as history), its records are
// read, its references are in place.
// Returns kOk or kPoolExhausted.  (No distance reaches beyond the window before
// the chunk: a code names 32768 at most.)
template <int LB, int NT>
__device__ __forceinline__ int32_t expand_tokens(CtaSmem<LB, NT>* S, const PagePool& pool, uint32_t n,
                                                 bool zero_window) {
  constexpr uint32_t kWin = CtaSmem<LB, NT>::kWin;
  const uint32_t tid = threadIdx.x;
  const uint64_t o = S->c.o;
  const uint64_t base = o & ~(uint64_t)(kWin - 1);  // positions below are relative to this
  const uint32_t rel0 = (uint32_t)(o - base);
  uint32_t lo = rel0;          // next position to write
  uint32_t b0 = 0;             // first slot of the batch
  uint32_t bpos = rel0, bend;  // positions of the batch
  uint32_t pos[kTokPer], len[kTokPer], rec[kTokPer], par = 0;
  if (tid < kWin / 16) (&S->bm[0][0])[tid] = 0;
  if (tid == 0) {
    S->c.carry_len = S->c.mark_max = 0;
  }
  cta_sync();
  // rec: what the slot puts at its position, a literal or a match's record
  // (length and distance - 1)
  auto load_batch = [&]() {
    const uint32_t i = b0 + kTokPer * tid;
    uint32_t sum = 0, prev = 0, next = 0;
    uint2 t = make_uint2(0, 0);
    if (i < n) {
      t = *reinterpret_cast<const uint2*>(S->tok + i);
      prev = i ? S->tok[i - 1] : 0u;
      next = S->tok[i + kTokPer];
    }
    const uint32_t val[kTokPer + 1] = {t.x & 0xFFFFu, t.x >> 16, t.y & 0xFFFFu, t.y >> 16, next};
#pragma unroll
    for (uint32_t k = 0; k < kTokPer; k++) {
      const bool match = val[k] & kTokMatch;
      len[k] = match ? val[k] & 0x1FFu : (prev & kTokMatch ? 0u : 1u);
      if (i + k >= n) len[k] = 0;
      rec[k] = match ? len[k] << 16 | val[k + 1] : val[k];
      prev = val[k];
      pos[k] = sum;
      sum += len[k];
    }
    uint32_t ta;
    const uint32_t a = cta_scan(S, par, sum, ta);
    par ^= 1;
#pragma unroll
    for (uint32_t k = 0; k < kTokPer; k++) pos[k] += bpos + a;
    bend = bpos + ta;
  };
  load_batch();
  for (uint32_t turn = 0;; turn ^= 1) {
    uint32_t* const stage = S->stage[turn];
    uint32_t* const bm = S->bm[turn];
    const uint32_t wbase = lo & ~(kWin - 1), wend = wbase + kWin;
    if (!cta_page(S, pool, base + wbase)) return kPoolExhausted;
    // (the thread that wrote it in the window before sees it in time, which is
    // enough for the vote)
    uint32_t any_match = S->c.carry_len;
    for (;;) {
      // the batch's tokens that start in this window
#pragma unroll
      for (uint32_t k = 0; k < kTokPer; k++) {
        const uint32_t q = pos[k] - wbase;
        if (len[k] && pos[k] >= lo && q < kWin) {
          stage[q] = rec[k];
          if (len[k] > 1) {
            atomicOr(&bm[q >> 5], 1u << (q & 31));
            any_match = 1;
          }
        }
      }
      if (bend >= wend || b0 + kTokPer * NT >= n) break;
      b0 += kTokPer * NT;
      bpos = bend;
      load_batch();
    }
    const bool matches = cta_sync_or(any_match != 0);
    const uint32_t hi = min(wend, bend) - wbase, l0 = lo - wbase;
    uint16_t* page = pool.data + (size_t)S->c.page_cur * kPageEntries +
                     ((uint32_t)(base + wbase) & (kPageEntries - 1));
    // this thread's positions: e0 .. e0 + 7
    const uint32_t e0 = kWinPer * tid;
    uint32_t st[kWinPer];  // a position's value, or (bit 31) a reference into the window
    {
      const uint4 a = reinterpret_cast<const uint4*>(stage)[2 * tid];
      const uint4 b = reinterpret_cast<const uint4*>(stage)[2 * tid + 1];
      st[0] = a.x, st[1] = a.y, st[2] = a.z, st[3] = a.w;
      st[4] = b.x, st[5] = b.y, st[6] = b.z, st[7] = b.w;
    }
    if (matches) {
      const int lane = tid & 31;
      const int32_t page_off = (int32_t)((uint32_t)(base + wbase) & (kPageEntries - 1));
      const uint16_t* pprev = pool.data + (size_t)S->c.page_prev * kPageEntries + kPageEntries;
      const uint16_t* pcur = pool.data + (size_t)S->c.page_cur * kPageEntries;
      const int64_t wabs = (int64_t)(base + wbase);
      const int32_t c_ms = S->c.carry_ms;
      const uint32_t c_len = S->c.carry_len, c_dist = S->c.carry_dist;
      // the last match start before e0: in this warp, else in the nine words
      // before the warp's (a match is at most 258 long), else the match that
      // reaches in from the window before
      uint32_t bits = (bm[tid >> 2] >> (8 * (tid & 3))) & 0xFFu;
      const int32_t own = (int32_t)e0 + 31 - __clz(bits | 1u);
      const uint32_t have = __ballot_sync(0xFFFFFFFFu, bits != 0);
      const int32_t wi = (int32_t)(tid >> 5) * 8 - 1 - lane;
      const uint32_t pw = lane < 9 && wi >= 0 ? bm[wi] : 0u;
      const uint32_t havep = __ballot_sync(0xFFFFFFFFu, pw != 0);
      const int32_t far = __shfl_sync(0xFFFFFFFFu, 32 * wi + 31 - __clz(pw | 1u), __ffs(havep | 0x80000000u) - 1);
      const uint32_t below = have & ((1u << lane) - 1);
      const int32_t near = __shfl_sync(0xFFFFFFFFu, own, 31 - __clz(below | 1u));
      const int32_t at = below ? near : (havep ? far : -1);
      int32_t ms = at >= 0 ? at : c_ms;
      uint32_t ml = c_len, md = c_dist;
      if (at >= 0) {
        const uint32_t d = stage[at];
        ml = d >> 16;
        md = (d & 0xFFFFu) + 1;
      }
      uint32_t cover = 0;  // bit i: position e0 + i is inside a match
      for (;;) {
        // positions [x0, x1) of this thread's eight that the match covers
        const uint32_t nx = bits ? (uint32_t)__ffs(bits) - 1 : kWinPer;
        const int32_t x0 = max(0, ms - (int32_t)e0);
        const int32_t x1 = min((int32_t)min(nx, hi - min(hi, e0)), ms + (int32_t)ml - (int32_t)e0);
        if (x0 < x1) {
          const uint32_t jj = (uint32_t)((int32_t)e0 + x0 - ms), cnt = (uint32_t)(x1 - x0);
          // every entry of an overlapping match maps to one before the match:
          // its place mod the distance (the quotient is exact for jj < 258)
          uint32_t r = jj;
          if (md < ml) r -= (uint32_t)__fdividef((float)jj + 0.5f, (float)md) * md;
          const int32_t s0 = ms - (int32_t)md + (int32_t)r, s1 = s0 + (int32_t)cnt - 1;
          const uint32_t mine = ((1u << x1) - 1) & ~((1u << x0) - 1);
          cover |= mine;
          const bool wrap = r + cnt > md;
          if (wrap && ms - (int32_t)md >= (int32_t)l0) {
            // round and round one stretch of this window
#pragma unroll
            for (uint32_t i = 0; i < kWinPer; i++)
              if ((mine >> i) & 1) {
                st[i] = 0x80000000u | (uint32_t)(ms - (int32_t)md + (int32_t)r);
                r = r + 1 == md ? 0u : r + 1;
              }
          } else if (!wrap && (s0 >= (int32_t)l0 || wabs + s1 < 0)) {
            // references into the window, or markers (zeros) before the chunk
            const bool ref = s0 >= (int32_t)l0;
            const uint32_t v0 = ref ? 0x80000000u | (uint32_t)s0
                                    : (uint32_t)((int64_t)(kMarkerBase + kWindow) + wabs + s0);
            const bool zero = !ref && zero_window;
#pragma unroll
            for (uint32_t i = 0; i < kWinPer; i++)
              if ((mine >> i) & 1) st[i] = zero ? 0u : v0 + i - (uint32_t)x0;
          } else if (!wrap && s1 < (int32_t)l0 && wabs + s0 >= 0 &&
                     (page_off + s0 >= 0) == (page_off + s1 >= 0)) {
            const uint16_t* from = (page_off + s0 >= 0 ? pcur : pprev) + (page_off + s0 - x0);
#pragma unroll
            for (uint32_t i = 0; i < kWinPer; i++)
              if ((mine >> i) & 1) st[i] = from[i];
          } else {
#pragma unroll
            for (uint32_t i = 0; i < kWinPer; i++) {
              if (!((mine >> i) & 1)) continue;
              const int32_t sr = ms - (int32_t)md + (int32_t)r;
              r = r + 1 == md ? 0u : r + 1;
              const int32_t q = page_off + sr;
              if (sr >= (int32_t)l0) st[i] = 0x80000000u | (uint32_t)sr;
              else if (wabs + sr >= 0) st[i] = (q >= 0 ? pcur : pprev)[q];
              else st[i] = zero_window ? 0u : (uint32_t)((int64_t)(kMarkerBase + kWindow) + wabs + sr);
            }
          }
        }
        if (!bits) break;
        bits &= bits - 1;
        ms = (int32_t)(e0 + nx);
        const uint32_t d = stage[ms];
        ml = d >> 16;
        md = (d & 0xFFFFu) + 1;
      }
      uint32_t left = 0;
#pragma unroll
      for (uint32_t i = 0; i < kWinPer; i++) left |= (cover >> i) & 1 ? st[i] : 0u;
      const bool any_ref = cta_sync_or(left >> 31);
      if (hi - 1 - e0 < kWinPer) {  // the last position's match may go on in the next window
        S->c.carry_ms = ms - (int32_t)kWin;
        S->c.carry_len = ms + (int32_t)ml > (int32_t)hi ? ml : 0u;
        S->c.carry_dist = md;
      }
      if (tid < kWin / 32) bm[tid] = 0;
      if (any_ref) {
        if (cover) {
          reinterpret_cast<uint4*>(stage)[2 * tid] = make_uint4(st[0], st[1], st[2], st[3]);
          reinterpret_cast<uint4*>(stage)[2 * tid + 1] = make_uint4(st[4], st[5], st[6], st[7]);
        }
        cta_sync();
        // A reference takes its source's value, or the source's own reference,
        // always further back: every thread follows its own to their ends,
        // and what it learns on the way shortens the others' paths.
        while (left >> 31) {
          left = 0;
#pragma unroll
          for (uint32_t i = 0; i < kWinPer; i++)
            if ((cover >> i) & 1 && st[i] >> 31) {
              st[i] = *(volatile uint32_t*)&stage[st[i] & 0xFFFFu];
              *(volatile uint32_t*)&stage[e0 + i] = st[i];
              left |= st[i];
            }
        }
        __syncwarp();
      }
    }
    // out to the page, eight entries per store
    {
      const uint4 v = make_uint4(__byte_perm(st[0], st[1], 0x5410), __byte_perm(st[2], st[3], 0x5410),
                                 __byte_perm(st[4], st[5], 0x5410), __byte_perm(st[6], st[7], 0x5410));
      const bool full = e0 >= l0 && e0 + kWinPer <= hi;
      if (full) {
        *reinterpret_cast<uint4*>(page + e0) = v;
      } else {
#pragma unroll
        for (uint32_t i = 0; i < kWinPer; i++)
          if (e0 + i >= l0 && e0 + i < hi) page[e0 + i] = (uint16_t)st[i];
      }
      if (matches && !zero_window) {
        uint32_t mk = 0;
        if ((v.x | v.y | v.z | v.w) & 0x80008000u) {
#pragma unroll
          for (uint32_t i = 0; i < kWinPer; i++)
            if (e0 + i >= l0 && e0 + i < hi && (st[i] & 0x8000u)) mk = e0 + i + 1;
        }
        if (__any_sync(0xFFFFFFFFu, mk != 0)) {
          mk = __reduce_max_sync(0xFFFFFFFFu, mk);
          if ((tid & 31) == 0) atomicMax(&S->c.mark_max, wbase + mk);
        }
      }
    }
    lo = wbase + hi;
    if (bend <= wend) {  // the batch is used up
      b0 += kTokPer * NT;
      if (b0 >= n) break;
      bpos = bend;
      load_batch();
      // only the distance of the match before is left: no position, so no window
      // (at a page's end it would take a page that gets no entry)
      if (bend == bpos) break;
    }
  }
  cta_sync();
  if (tid == 0) {
    S->c.o = base + lo;
    if (S->c.mark_max) S->c.marker_end = base + S->c.mark_max;
  }
  return kOk;
}

// The pool ran out in a round of n slots that ends at new_pos: move S->c.o to the
// entries written and S->c.pos by the same share of the round, which the larger pool
// is sized by.  (Apart from expand_tokens, whose loop is 5 % slower on byte runs
// when it keeps count itself.)
template <int LB, int NT>
__device__ __noinline__ void cta_progress(CtaSmem<LB, NT>* S, uint32_t n, uint64_t new_pos) {
  const uint32_t tid = threadIdx.x;
  if (tid == 0) S->c.mark_max = 0;
  cta_sync();
  uint32_t sum = 0;  // entries of the round
  for (uint32_t i = tid; i < n; i += NT) {
    const uint32_t v = S->tok[i];
    sum += v & kTokMatch ? v & 0x1FFu : (i && S->tok[i - 1] & kTokMatch ? 0u : 1u);
  }
  atomicAdd(&S->c.mark_max, sum);
  cta_sync();
  const uint64_t at = (uint64_t)S->c.page_seq * kPageEntries;  // the page there was none for
  if (tid == 0 && at > S->c.o) {
    const float part = (float)(uint32_t)(at - S->c.o) / (float)S->c.mark_max;
    S->c.pos += (uint32_t)(fminf(part, 1.f) * (float)(uint32_t)(new_pos - S->c.pos));
    S->c.o = at;
  }
}

// The body of one Huffman-coded block, tables in place.  On return (after a
// barrier) S->c holds the new position and entry count, status, synced (at
// the successor's sync start) or passed (went by the successor's start).
template <int LB, int NT>
__device__ __forceinline__ void cta_block(const uint8_t* __restrict__ in, CtaSmem<LB, NT>* S,
                                          const PagePool& pool, bool zero_window) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  constexpr uint32_t kTokCap = CtaSmem<LB, NT>::kTokCap;
  const uint32_t tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  uint32_t rcap = kRangeMax;
  for (;;) {
    // every thread computes the round's geometry from the shared state
    const uint64_t pos = S->c.pos, limit = S->c.limit_words, trunc = S->c.trunc_words;
    const uint64_t target = S->c.sync_target;
    const uint64_t w0 = pos >> 5;
    if (target == pos || w0 + 4 > limit) {
      cta_sync();
      if (tid == 0) {
        if (target == pos) S->c.synced = 1;
        else S->c.status = w0 + 4 > trunc ? kTruncated : kOvershoot;
      }
      break;
    }
    uint64_t end = (limit - 3) * 32;  // symbols start below this
    if (target != kNoStop && target > pos && target < end) end = target;
    const uint64_t likely = S->c.stop_lo > pos && S->c.stop_lo < end ? S->c.stop_lo : end;
    const uint64_t want = ((likely - pos) / NT + 32) & ~31ull;
    const uint32_t r = (uint32_t)max((uint64_t)kRangeMin, min(want, (uint64_t)rcap));
    const uint32_t p0 = (uint32_t)(pos & 31);
    const uint64_t span = end - pos;
    const uint32_t pend = p0 + (uint32_t)min(span, (uint64_t)r * NT);
    const uint32_t lanes = (pend - p0 + r - 1) / r;
    const uint32_t* base = in32 + w0;
    // 1. from the guessed starts (a range cut off by a stop keeps the end it had: its own start)
    const bool active = tid < lanes;
    if (active) {
      S->start[tid] = S->end[tid] = p0 + tid * r;
      walk_range<LB, NT>(S, base, p0 + tid * r, r, min(p0 + tid * r + r, pend), tid, tid > 0, false);
    }
    __syncwarp();
    // 2. from the end of the range before, until nothing moves.  The ranges to
    // walk again go to the first threads, so that few of them are few warps.
    uint32_t last = kNone;  // range that holds the end of the block (kNone: not in this round)
    for (;;) {
      cta_sync();
      const uint32_t st = active ? S->start[tid] : 0u, inf = active ? S->info[tid] : 0u;
      const uint32_t s1 = active && tid ? S->end[tid - 1] : st;
      const bool need = active && (s1 != st || (inf & kInfoOn));
      const uint32_t nb = __ballot_sync(0xFFFFFFFFu, need);
      const uint32_t tb = __ballot_sync(0xFFFFFFFFu, (inf / kInfoTerm) & 3);
      if (lane == 0) {
        S->need[warp] = nb;
        S->term[warp] = tb;
      }
      if (need) S->start[tid] = s1;
      cta_sync();
      const uint32_t mn = lane < NT / 32 ? S->need[lane] : 0u;
      const uint32_t mt = lane < NT / 32 ? S->term[lane] : 0u;
      const uint32_t bn = __ballot_sync(0xFFFFFFFFu, mn != 0), bt = __ballot_sync(0xFFFFFFFFu, mt != 0);
      const int wn = __ffs(bn | 0x80000000u) - 1, wt = __ffs(bt | 0x80000000u) - 1;
      const uint32_t first_need = 32u * wn + __ffs(__shfl_sync(0xFFFFFFFFu, mn, wn)) - 1;
      const uint32_t first_term = 32u * wt + __ffs(__shfl_sync(0xFFFFFFFFu, mt, wt)) - 1;
      last = bt ? first_term : kNone;
      if (!bn || last < first_need) break;
      uint32_t upto = __popc(mn);
#pragma unroll
      for (int d = 1; d < NT / 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, upto, d);
        if (lane >= d) upto += u;
      }
      const uint32_t before = __shfl_sync(0xFFFFFFFFu, upto - __popc(mn), warp);
      const uint32_t n_need = __shfl_sync(0xFFFFFFFFu, upto, NT / 32 - 1);
      if (need) S->list[before + __popc(nb & ((1u << lane) - 1))] = (uint16_t)tid;
      cta_sync();
      if (tid < n_need) {
        const uint32_t id = S->list[tid], f = p0 + id * r;
        walk_range<LB, NT>(S, base, f, r, min(f + r, pend), id, false, true);
      }
      __syncwarp();
    }
    // 3. places in the token list; ranges beyond its capacity wait for the next round
    const uint32_t used = last != kNone ? last + 1 : lanes;
    const bool in_use = tid < used;
    uint32_t ts;
    const uint32_t my_info = in_use ? S->info[tid] : 0u, my_start = in_use ? S->start[tid] : 0u;
    const uint32_t my_slots = my_info & 0xFFFFu, my_term = (my_info / kInfoTerm) & 3;
    const uint32_t slot0 = cta_scan(S, 0, my_slots, ts);
    if (ts > kTokCap) {
      const uint32_t fit = (uint32_t)cta_sync_count(in_use && slot0 + my_slots <= kTokCap);
      if (tid == fit) {
        S->c.round_slots = slot0;
        S->c.round_pos = my_start;  // = the end of range fit - 1
      }
      if (tid == 0) {
        S->c.round_lanes = fit;
        S->c.round_kind = kTermNone;
      }
      // shorter ranges from here on: about nine tenths of the list
      rcap = max(kRangeMin, min(rcap, (uint32_t)((uint64_t)r * kTokCap / ts * 9 / 10)) & ~31u);
    } else if (tid == used - 1) {
      S->c.round_slots = ts;
      S->c.round_lanes = used;
      S->c.round_kind = my_term;
      S->c.round_pos = my_term ? S->term_pos[tid] : S->end[tid];
    }
    cta_sync();
    const uint32_t n_lanes = S->c.round_lanes, n_slots = S->c.round_slots;
    const uint32_t kind = S->c.round_kind;
    const uint64_t new_pos = w0 * 32 + S->c.round_pos;
    if (kind == kTermBad) {
      cta_sync();
      if (tid == 0) S->c.status = kBadDeflate;
      break;
    }
    if (tid < n_lanes) write_tokens<LB, NT>(S, base, my_start, my_slots, S->tok + slot0);
    cta_sync();
    // 4. expansion
    if (n_slots) {
      const int32_t st = expand_tokens<LB, NT>(S, pool, n_slots, zero_window);
      if (st != kOk) {
        cta_sync();
        cta_progress<LB, NT>(S, n_slots, new_pos);
        if (tid == 0) S->c.status = st;
        break;
      }
    }
    const bool passed = S->c.passed_bit < new_pos;
    cta_sync();
    if (tid == 0) {
      S->c.pos = new_pos;
      if (kind == kTermNone && passed && new_pos != target) S->c.passed = 1;
    }
    cta_sync();
    if (kind == kTermEob || S->c.passed) break;
  }
  cta_sync();
}

// A stored block's bytes to the chunk's pages, four entries per thread.
template <int LB, int NT>
__device__ __forceinline__ void cta_stored(const uint8_t* __restrict__ in, CtaSmem<LB, NT>* S,
                                           const PagePool& pool) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  uint64_t byte = S->c.pos >> 3, o = S->c.o;
  uint32_t left = S->c.stored_len;
  bool ok = true;
  while (left) {
    if (!cta_page(S, pool, o)) {
      ok = false;
      break;
    }
    const uint32_t q = (uint32_t)o & (kPageEntries - 1);
    const uint32_t n = min(left, kPageEntries - q);
    uint16_t* dst = pool.data + (size_t)S->c.page_cur * kPageEntries;
    // groups of 4 entries aligned to 4; the first and last may be partial
    for (uint32_t g = (q & ~3u) + 4 * threadIdx.x; g < q + n; g += 4 * NT) {
      if (g >= q && g + 4 <= q + n) {
        const uint64_t a = byte + (g - q);
        const uint32_t v = __funnelshift_r(in32[a >> 2], in32[(a >> 2) + 1], 8 * ((uint32_t)a & 3));
        *reinterpret_cast<uint2*>(dst + g) =
            make_uint2(__byte_perm(v, 0, 0x4140), __byte_perm(v, 0, 0x4342));
      } else {
        for (uint32_t i = max(g, q); i < min(g + 4, q + n); i++) dst[i] = in[byte + (i - q)];
      }
    }
    byte += n;
    o += n;
    left -= n;
  }
  cta_sync();
  if (threadIdx.x == 0) {
    S->c.pos = byte * 8;
    S->c.o = o;
    if (!ok) S->c.status = kPoolExhausted;
  }
  cta_sync();
}

// what the chunk does next
enum : int32_t {
  kActDone = 0,     // the chunk is finished (status)
  kActResume,       // the same block goes on, tables in place
  kActHeader,       // a block header at pos
  kActTable,        // a sync start: read the header at table_bit, then go on at pos
  kActFixed,        // a sync start in a fixed block
  kActStored,       // copy stored_len bytes at pos
  kActBlock,        // read the code lengths (dynamic), build the tables, decode the block
};

// start bit a predecessor must reach to hand over to chunk k
__device__ __forceinline__ uint64_t handover_bit(const ChunkDesc& k) {
  return (k.flags & kChunkMemberFirst) ? k.limit_bit * 8 : k.lo_bit;
}

// the reader may run up to the abort bit (moved on by every extension)
__device__ __forceinline__ void cta_set_limit(CtaCtl& c) {
  c.limit_words = (c.abort_bit != kNoStop && c.abort_bit / 32 + 5 < c.trunc_words)
                      ? c.abort_bit / 32 + 5
                      : c.trunc_words;
}

// move on past successor c.next (a phantom) to nx, the chunk after it
__device__ __forceinline__ void cta_extend(CtaCtl& c, const ChunkDesc* descs, uint32_t nx) {
  if (nx == kNoChunk) {
    c.stop_lo = kNoStop;
    c.abort_bit = kNoStop;
  } else {
    c.stop_lo = handover_bit(descs[nx]);
    if (c.abort_bit != kNoStop) c.abort_bit = c.stop_lo + c.slack;
  }
  c.next = nx;
  c.extends++;
  cta_set_limit(c);
}

// At a block boundary (or after going by a successor mid-block): stop, or
// what to read next.  Thread 0 only.
__device__ __noinline__ int32_t cta_boundary(CtaCtl& c, const ChunkDesc* descs, const PagePool& pool) {
  const bool confirmed = (c.flags & (kChunkMemberFirst | kChunkConfirmed)) != 0;
  const bool resume_now = c.resume != 0;
  c.resume = 0;
  const uint64_t bitpos = c.pos;
  while (!resume_now && bitpos >= c.stop_lo) {
    // A block boundary past the successor's start range means that start
    // was a phantom: decode on to the start after it (the consumer's
    // re-decode from the confirmed boundary, chunk_fetcher.rs:855).
    if (c.next == kNoChunk) return kActDone;
    if (c.extends >= kMaxExtends && !confirmed) return kActDone;
    const ChunkDesc nx = descs[c.next];
    if (nx.flags & kChunkMemberFirst) return kActDone;
    // the successor's CTA may have moved its start to a later candidate
    // (in-kernel retry) since this chunk's stop was set: read its range
    // afresh and keep decoding while still before it.  A stale or torn
    // read only costs a repair: the host walk checks every handover.
    const volatile ChunkDesc* vx = descs + c.next;
    const uint64_t nx_lo = vx->lo_bit, nx_start = vx->start_bit;
    if (bitpos < nx_lo) {
      c.stop_lo = nx_lo;
      if (c.abort_bit != kNoStop) c.abort_bit = c.stop_lo + c.slack;
      cta_set_limit(c);
      break;
    }
    // a sync start is taken over only mid-block, at its exact symbol start
    // (cta_block); a block boundary at or past it means this chunk went by it
    if (!(nx.flags & kChunkSync) && bitpos <= nx_start) return kActDone;
    cta_extend(c, descs, nx.next);
  }
  if (resume_now) {
    // successors whose start this chunk is already past, mid-block
    while (c.next != kNoChunk && (confirmed || c.extends < kMaxExtends)) {
      if ((descs[c.next].flags & kChunkMemberFirst) ||
          ((const volatile ChunkDesc*)(descs + c.next))->start_bit >= bitpos)
        break;
      cta_extend(c, descs, descs[c.next].next);
    }
  }
  if (bitpos > c.abort_bit) {
    c.status = kOvershoot;
    return kActDone;
  }
  if (bitpos + 3 > c.in_end * 8) {
    c.status = kTruncated;
    return kActDone;
  }
  if (resume_now) return kActResume;
  if (c.in_sync_block) {
    c.in_sync_block = 0;
    if (c.table_bit) {
      c.blk_hdr = c.table_bit;
      return kActTable;
    }
    c.bfinal = 0;
    c.btype = 1;
    c.blk_hdr = 0;
    return kActFixed;
  }
  c.blk_hdr = bitpos;
  if (pool.blocks) {
    const uint32_t k = atomicAdd(pool.n_blocks, 1u);
    if (k < pool.blocks_cap) pool.blocks[k] = BlockRec{bitpos, c.o, c.cid, c.gen};
  }
  return kActHeader;
}

// Where this block may hand over mid-block.  The successor's sync start can
// be taken over only in the state it assumes: inside its block (same header),
// or inside a non-final fixed block for a fixed sync start.  Any successor
// whose start goes by mid-block is a phantom (real starts are block
// boundaries or sync starts reached exactly): the decode moves on past it.
__device__ __forceinline__ void cta_targets(CtaCtl& c, const ChunkDesc* descs, bool sync) {
  c.sync_target = c.passed_bit = kNoStop;
  if (!sync || c.next == kNoChunk) return;
  const ChunkDesc& nx = descs[c.next];
  if (nx.flags & kChunkSync) {
    const bool same = nx.table_bit ? (c.blk_hdr == nx.table_bit) : (c.btype == 1 && !c.bfinal);
    if (same) c.sync_target = nx.start_bit;
  }
  const bool confirmed = (c.flags & (kChunkMemberFirst | kChunkConfirmed)) != 0;
  if (!(nx.flags & kChunkMemberFirst) && (confirmed || c.extends < kMaxExtends))
    c.passed_bit = ((const volatile ChunkDesc*)(descs + c.next))->start_bit;
}

// One warp: the boundary's decision and the start of the header it leads to
// (a dynamic block's up to its precode).
template <int LB, int NT>
__device__ __noinline__ void cta_header(const uint8_t* __restrict__ in, const ChunkDesc* descs,
                                        CtaSmem<LB, NT>* S, const PagePool& pool, bool sync, int lane) {
  CtaCtl& c = S->c;
  int32_t act = kActDone;
  if (lane == 0) act = cta_boundary(c, descs, pool);
  act = __shfl_sync(0xFFFFFFFFu, act, 0);
  __syncwarp();
  int32_t status = kOk;
  bool fixed = act == kActFixed;
  const bool table = act == kActTable;
  if (act == kActHeader || table) {
    // 128 bits from the header on (zeros past the input)
    const uint64_t start = table ? c.table_bit : c.pos, w0 = start >> 5;
    const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
    const uint32_t w = lane < 5 && w0 + lane < c.trunc_words ? in32[w0 + lane] : 0u;
    const uint32_t wn = __shfl_down_sync(0xFFFFFFFFu, w, 1);
    const uint32_t b = __funnelshift_r(w, wn, (uint32_t)(start & 31));
    const uint64_t lo = (uint64_t)__shfl_sync(0xFFFFFFFFu, b, 1) << 32 | __shfl_sync(0xFFFFFFFFu, b, 0);
    const uint64_t hi = (uint64_t)__shfl_sync(0xFFFFFFFFu, b, 3) << 32 | __shfl_sync(0xFFFFFFFFu, b, 2);
    const uint32_t btype = (uint32_t)(lo >> 1) & 3;
    uint64_t pos = start + 3;
    uint32_t stored = 0, nlen = 0, ndist = 0;
    if (btype == 3 || (btype == 0 && table)) {
      status = kBadDeflate;
    } else if (btype == 0) {
      // stored block: byte-align, LEN/NLEN
      pos = (pos + 7) & ~7ull;
      const uint32_t sz = (uint32_t)(lo >> (pos - start));
      stored = sz & 0xFFFF;
      pos += 32;
      const uint64_t byte = pos >> 3;
      if (byte > c.in_end) status = kTruncated;
      else if (stored != (~(sz >> 16) & 0xFFFFu)) status = kBadDeflate;
      else if (byte + stored > c.in_end) status = kTruncated;
      act = kActStored;
    } else if (btype == 1) {
      fixed = true;
    } else {
      const uint32_t h = (uint32_t)(lo >> 3);
      nlen = 257 + (h & 31);
      ndist = 1 + ((h >> 5) & 31);
      const uint32_t ncl = 4 + ((h >> 10) & 15);
      if (nlen > 286 || ndist > 30) status = kBadDeflate;
      // code-length code lengths: 3 bits each from bit 17 on
      const uint64_t pb = lo >> 17 | hi << 47;
      if (lane < 19)
        S->pre_lens[c_cl_order[lane]] =
            (uint32_t)lane < ncl ? (uint8_t)((pb >> (3 * lane)) & 7) : (uint8_t)0;
      __syncwarp();
      if (status == kOk && !index_code(S->pre_lens, 19, &S->lit, S->lit_ent, lane, pre_entry))
        status = kBadDeflate;
      pos = start + 17 + 3 * ncl;
      act = kActBlock;
    }
    __syncwarp();
    if (lane == 0) {
      c.bfinal = (uint32_t)lo & 1;
      c.btype = btype;
      c.hdr_pos = pos;
      c.hdr_move = !table;
      if (!table) c.pos = pos;
      c.nlen = nlen;
      c.ndist = ndist;
      c.stored_len = stored;
      if (btype == 2) c.fixed_tables = 0;  // the precode took their place
    }
  }
  if (fixed) {
    act = kActBlock;
    if (!c.fixed_tables) {
      // fixed Huffman (RFC 1951 3.2.6): litlen 0..287, then 32 distance codes
      for (int s = lane; s < 320; s += 32)
        S->lens[s] = s < 144 ? 8 : (s < 256 ? 9 : (s < 280 ? 7 : (s < 288 ? 8 : 5)));
      if (lane == 0) {
        c.nlen = 288;
        c.ndist = 32;
      }
    }
  }
  __syncwarp();
  if (lane == 0) {
    if (status != kOk) {
      c.status = status;
      act = kActDone;
    }
    c.act = act;
    if (act == kActBlock || act == kActResume) cta_targets(c, descs, sync);
  }
}

// Decode one chunk; its state is in S->c (prepared by cta_begin).
template <int LB, int NT>
__device__ __forceinline__ void cta_decode_chunk(const uint8_t* __restrict__ in, const ChunkDesc* descs,
                                                 ChunkResult* res, CtaSmem<LB, NT>* S,
                                                 const PagePool& pool, bool sync) {
  const int tid = threadIdx.x;
  CtaCtl& c = S->c;
  const bool zero_window = (c.flags & kChunkMemberFirst) != 0;
  for (;;) {
    if (tid < 32) cta_header<LB, NT>(in, descs, S, pool, sync, tid);
    cta_sync();
    const int32_t act = c.act;
    if (act == kActDone) break;
    if (act == kActStored) {
      cta_stored<LB, NT>(in, S, pool);
    } else {
      if (act == kActBlock && !(c.btype == 1 && c.fixed_tables)) {
        int32_t st = c.btype == 2 ? cta_read_lens<LB, NT>(in, S, c.hdr_move != 0) : kOk;
        if (st == kOk && !cta_build_tables<LB, NT>(S)) st = kBadDeflate;
        if (tid == 0) {
          c.fixed_tables = st == kOk && c.btype == 1;
          if (st != kOk) c.status = st;
        }
        cta_sync();
        if (st != kOk) break;
      }
      cta_block<LB, NT>(in, S, pool, zero_window);
    }
    if (c.status != kOk || c.synced) break;
    const bool passed = c.passed != 0, fin = c.bfinal != 0;
    cta_sync();
    if (tid == 0) {
      if (passed) {
        c.passed = 0;
        c.resume = 1;
        cta_extend(c, descs, descs[c.next].next);
      } else {
        c.n_blocks++;
        c.final_block = fin;
      }
    }
    if (!passed && fin) break;
  }
  cta_sync();
  if (tid == 0) {
    if (c.status == kOk && c.pos > c.in_end * 8) c.status = kTruncated;
    res->end_bit = c.pos;
    res->out_len = c.o;
    res->marker_end = c.marker_end;
    // the page of the last entry, and the one before it
    res->last_page = c.o ? c.page_cur : kNoPage;
    res->prev_page = c.o ? c.page_prev : kNoPage;
    res->n_pages = c.n_pages;
    res->n_blocks = c.n_blocks;
    res->status = c.status;
    res->final_block = (int32_t)c.final_block;
    res->gen = c.gen;
    res->sync_end = c.synced;
    res->end_hdr_bit = c.synced ? c.blk_hdr : 0;
  }
  cta_sync();
}

// Thread 0: the state a chunk's decode begins with.
__device__ __forceinline__ void cta_begin(CtaCtl& c, const ChunkDesc& d, uint32_t cid, uint32_t gen) {
  c.pos = d.start_bit;
  c.o = 0;
  c.stop_lo = d.stop_lo;
  c.abort_bit = d.abort_bit;
  c.slack = d.abort_bit != kNoStop ? d.abort_bit - d.stop_lo : 0;
  c.in_end = d.in_end;
  c.trunc_words = (d.in_end * 8 + 31) / 32 + 5;
  c.table_bit = d.table_bit;
  c.blk_hdr = 0;
  c.marker_end = 0;
  c.next = d.next;
  c.flags = d.flags;
  c.cid = cid;
  c.gen = gen;
  c.n_blocks = c.extends = c.final_block = c.synced = c.passed = c.resume = 0;
  c.in_sync_block = (d.flags & kChunkSync) != 0;
  c.spec = d.limit_bit > d.lo_bit;
  c.status = kOk;
  c.page_cur = c.page_prev = kNoPage;
  c.page_seq = 0;
  c.n_pages = 0;
  c.bfinal = c.btype = 0;
  cta_set_limit(c);
}

}  // namespace gzgpu
