// block_cta.cuh -- one CTA decodes one chunk (page history).
//
// Block body.  A Huffman-coded block is decoded in rounds of up to
// kCtaThreads bit ranges of `r` bits each, one range per thread:
//   1. every thread decodes its range from a guessed start (its first bit).
//      Prefix codes resynchronise: a decode that starts off a symbol boundary
//      falls into step with the true one, so most ranges end at the right
//      bit although they started at a wrong one.
//   2. each range is decoded again from where the range before it ended, and
//      again while that end moves, until no start changes (or all ranges up
//      to one that met the end of the block agree).  By induction from the
//      first range, whose start is exact, the joined ranges are the serial
//      decode.  Each pass confirms at least one more range.
//   3. a block scan of the ranges' symbol counts gives each its place in the
//      round's token list (a literal: one slot; a match: length, then
//      distance), written in one more decode pass.
//   4. the tokens are expanded in windows of kWin output positions (see
//      expand_tokens), which leave as coalesced stores to the pages.
// What bounds a block is its serial chain of code lookups; the ranges cut
// that chain into up to 256 pieces.  Ranges of 512 bits end in step after a
// wrong start for 98 % of text, 88 % of byte runs and 59 % of noisy ramps
// (codes nearly all of one length), measured on zlib level 6 streams.
// Inflate kernel, before (one warp per chunk, steps of 64 bits decoded by the
// whole warp) and now: 64 MiB text 6.9 -> 1.0 ms, 12 MiB ramps 4.6 -> 0.9,
// 64 MiB byte runs 22 -> 2.0, 16 MiB of fixed codes 7.8 -> 0.31, a 4 KiB
// stream 0.195 -> 0.068.
#pragma once
#include <cstdint>

#include "common.cuh"
#include "huffman.cuh"
#include "inflate.cuh"

namespace gzgpu {

constexpr uint32_t kRangeMax = 512;   // bits per thread and round, at most
constexpr uint32_t kRangeMin = 64;    // and at least (more than the longest symbol's 48)
constexpr uint32_t kTokCap = 12288;   // token slots per round
constexpr uint32_t kWin = 2048;       // output positions expanded at a time (divides a page)
constexpr uint32_t kWinPer = kWin / kCtaThreads;
constexpr uint32_t kTokPer = 4;       // token slots per thread and batch
constexpr uint32_t kCtaDistBits = 9;  // distance LUT index bits
constexpr uint32_t kInWords = kCtaThreads * kRangeMax / 32 + 8;
constexpr uint32_t kNone = 0xFFFFFFFFu;

// table entry: [4:0] bits of the code and its extra bits, bit 5 = length code,
// bit 6 = not a literal, length or distance (end of block, or, by value:
// invalid, or not in the LUT), bit 7 = literal, [23:8] token value without the
// extra bits, [31:28] code length
enum : uint32_t { kEntLen = 0x20, kEntStop = 0x40, kEntLit = 0x80 };
enum : uint32_t { kStopEob = 0, kStopBad = 1, kStopLong = 2 };
constexpr uint32_t kTokMatch = 0x8000u;  // a match's first slot: flag and length

__device__ __forceinline__ uint32_t tok_lit_entry(uint32_t sym, uint32_t L) {
  if (sym < 256) return L << 28 | sym << 8 | kEntLit | L;
  if (sym == 256) return L << 28 | kStopEob << 8 | kEntStop | L;
  if (sym <= 285) {
    const uint32_t k = sym - 257;
    return L << 28 | (kTokMatch + c_len_base[k]) << 8 | kEntLen | (L + c_len_extra[k]);
  }
  return L << 28 | kStopBad << 8 | kEntStop | L;
}
__device__ __forceinline__ uint32_t tok_dist_entry(uint32_t sym, uint32_t L) {
  if (sym < 30) return L << 28 | (uint32_t)(c_dist_base[sym] - 1) << 8 | (L + c_dist_extra[sym]);
  return L << 28 | kStopBad << 8 | kEntStop | L;
}

// the chunk's state, written by thread 0 (or warp 0) and read by all after a barrier
struct CtaCtl {
  uint64_t pos, o;          // next input bit, entries written
  uint64_t stop_lo, abort_bit, slack, limit_words, trunc_words, in_end, table_bit;
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
  uint32_t build_ok[2];
  uint32_t page_cur, page_prev, page_seq, n_pages;
  uint32_t min_need[2], min_term[2];
  uint32_t round_slots, round_out, round_lanes, round_kind, round_pos;
  int32_t carry_ms;         // match reaching into the next window: start (relative to it)
  uint32_t carry_len, carry_dist;
  uint32_t any_match, bad_dist, mark_max;
};

template <int LB>
struct alignas(16) CtaSmem {
  uint32_t lit_lut[1 << LB];
  uint32_t dist_lut[1 << kCtaDistBits];
  uint16_t tok[kTokCap + 8];
  union {
    HeaderScratch h;                           // block header
    uint32_t in[kInWords + kInWords / 32 + 4]; // decode: the round's input words (padded by skew)
    struct {                                   // expansion
      uint32_t stage[kWin];
      uint32_t bm[kWin / 32];                  // match starts
      int32_t lastm[kWin / 32];                // last match start before each word's positions
    };
  };
  uint16_t lit_sorted[288], dist_sorted[32];
  uint16_t lit_count[16], lit_first[16], lit_offs[16];
  uint16_t dist_count[16], dist_first[16], dist_offs[16];
  uint16_t dist_next[16];
  uint32_t end[kCtaThreads];
  uint32_t scan_a[2][kCtaThreads / 32], scan_b[2][kCtaThreads / 32];
  CtaCtl c;
};

// word j of the round's input, skewed so that threads at the same place of
// their ranges read different banks
__device__ __forceinline__ uint32_t in_at(uint32_t j) { return j + (j >> 5); }

// exclusive prefix sums of a and b over the CTA; totals in ta, tb.  One
// barrier; `par` alternates between calls (0, 1, 0, ...).
template <int LB>
__device__ __forceinline__ void cta_scan2(CtaSmem<LB>* S, uint32_t par, uint32_t& a, uint32_t& b,
                                          uint32_t& ta, uint32_t& tb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = a, y = b;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, d), v = __shfl_up_sync(0xFFFFFFFFu, y, d);
    if (lane >= d) {
      x += u;
      y += v;
    }
  }
  if (lane == 31) {
    S->scan_a[par][warp] = x;
    S->scan_b[par][warp] = y;
  }
  __syncthreads();
  uint32_t pa = 0, pb = 0;
  ta = tb = 0;
#pragma unroll
  for (int w = 0; w < kCtaThreads / 32; w++) {
    const uint32_t u = S->scan_a[par][w], v = S->scan_b[par][w];
    if (w < warp) {
      pa += u;
      pb += v;
    }
    ta += u;
    tb += v;
  }
  a = pa + x - a;
  b = pb + y - b;
}

// Codes longer than the LUT, or invalid: canonical search.  Returns the entry.
template <int LB>
__device__ __noinline__ uint32_t long_entry(const CtaSmem<LB>* S, uint32_t x, bool dist) {
  const uint32_t rev = __brev(x) >> 17;  // 15 code bits, first bit = MSB
  const uint16_t* count = dist ? S->dist_count : S->lit_count;
  const uint16_t* first = dist ? S->dist_first : S->lit_first;
  for (int L = 1; L <= 15; L++) {
    const uint32_t idx = (rev >> (15 - L)) - first[L];
    if (idx < count[L])
      return dist ? tok_dist_entry(S->dist_sorted[S->dist_offs[L] + idx], (uint32_t)L)
                  : tok_lit_entry(S->lit_sorted[S->lit_offs[L] + idx], (uint32_t)L);
  }
  return kStopBad << 8 | kEntStop;
}

// What one range decoded to.  A range that meets the end of the block or an
// invalid code has term set; slots and outs then count up to there.
struct RangeOut {
  uint32_t end, slots, outs, term, term_pos;
};
enum : uint32_t { kTermNone = 0, kTermEob = 1, kTermBad = 2 };

// Decode the symbols that start in [p, e) (bits relative to the staged
// input).  One table lookup per iteration: a literal or a length code, or the
// distance code of the length just read, so threads at literals and threads
// inside matches run the same instructions.  guess: p may be no symbol
// boundary; decode on past an end of block or an invalid code (from its next
// bit) to find a likely end for the range.  kTok: write the tokens.
template <int LB, bool kTok>
__device__ __forceinline__ void walk_range(const CtaSmem<LB>* S, uint32_t p, uint32_t e, bool guess,
                                           RangeOut& r, uint16_t* tok) {
  constexpr uint32_t LM = (1u << LB) - 1, DM = (1u << kCtaDistBits) - 1;
  uint32_t j = p >> 5, sh = p & 31;
  uint32_t w0 = S->in[in_at(j)], w1 = S->in[in_at(j + 1)], w2 = S->in[in_at(j + 2)];
  j += 3;
  uint32_t slots = 0, outs = 0, is_len = 0;
  uint32_t term = kTermNone, t_slots = 0, t_outs = 0, t_pos = 0;
  while (is_len || p < e) {
    const uint32_t x = __funnelshift_r(w0, w1, sh);
    const uint32_t* t = is_len ? S->dist_lut + (x & DM) : S->lit_lut + (x & LM);
    uint32_t ent = *t;
    if (ent & kEntStop) {
      if (((ent >> 8) & 3) == kStopLong) ent = long_entry<LB>(S, x, is_len != 0);
      if (ent & kEntStop) {
        if (kTok) break;  // the range's last symbol is the end of the block
        if (term == kTermNone) {
          const bool eob = ((ent >> 8) & 3) == kStopEob;
          term = eob ? kTermEob : kTermBad;
          t_slots = slots;
          t_outs = outs;
          t_pos = p + (eob ? ent & 31 : 0u);
        }
        if (!guess) break;
        ent = 1;  // go on at the next bit
      }
    }
    const uint32_t n = ent & 31;
    const uint32_t v = (ent >> 8) + ((x & ~(0xFFFFFFFFu << n)) >> (ent >> 28));
    if (kTok) tok[slots] = (uint16_t)v;
    is_len = ent & kEntLen;
    slots++;
    outs += is_len ? (v & 0x1FFu) : (ent >> 7) & 1u;
    p += n;
    sh += n;
    if (sh >= 32) {
      sh -= 32;
      w0 = w1;
      w1 = w2;
      w2 = S->in[in_at(j)];
      j++;
    }
  }
  r.end = p;
  r.term = term;
  r.slots = term ? t_slots : slots;
  r.outs = term ? t_outs : outs;
  r.term_pos = t_pos;
}

// Both code tables from h.lens (whole CTA).  Warp 0 sorts the
// literal/length code, warp 1 the distance code, all threads fill the LUTs.
// Distance lengths sit at lens + 288.
template <int LB>
__device__ __forceinline__ bool cta_build_tables(CtaSmem<LB>* S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < 2) {
    bool ok;
    if (warp == 0)
      ok = canon_build(S->h.lens, (int)S->c.nlen, S->lit_count, S->lit_first, S->lit_offs,
                       S->lit_sorted, S->h.next, lane);
    else
      ok = canon_build(S->h.lens + 288, (int)S->c.ndist, S->dist_count, S->dist_first, S->dist_offs,
                       S->dist_sorted, S->dist_next, lane);
    if (lane == 0) S->c.build_ok[warp] = ok;
  }
  __syncthreads();
  if (!S->c.build_ok[0] || !S->c.build_ok[1]) return false;
  for (uint32_t i = threadIdx.x; i < (1u << LB); i += kCtaThreads) {
    const uint32_t e = lut_entry<LB>(i, S->lit_count, S->lit_first, S->lit_offs, S->lit_sorted,
                                     tok_lit_entry);
    S->lit_lut[i] = e ? e : kStopLong << 8 | kEntStop;
  }
  for (uint32_t i = threadIdx.x; i < (1u << kCtaDistBits); i += kCtaThreads) {
    const uint32_t e = lut_entry<(int)kCtaDistBits>(i, S->dist_count, S->dist_first, S->dist_offs,
                                                    S->dist_sorted, tok_dist_entry);
    S->dist_lut[i] = e ? e : kStopLong << 8 | kEntStop;
  }
  __syncthreads();
  return true;
}

// Make the page of the window at chunk position w0 current (thread 0
// allocates, then a barrier).  Windows are visited in order and never cross a
// page.  False when the pool is exhausted.
template <int LB>
__device__ __forceinline__ bool cta_page(CtaSmem<LB>* S, const PagePool& pool, uint64_t w0) {
  const uint32_t s = (uint32_t)(w0 >> 16);
  if (S->c.page_cur != kNoPage && S->c.page_seq == s) return true;
  __syncthreads();
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
  __syncthreads();
  return S->c.page_cur != kNoPage;
}

// Expand a round's tokens (slots [0, n), total_out entries) after the
// chunk's entry position S->c.o.  Output goes in windows of kWin positions
// aligned to kWin, so a window lies in one page.  Batches of kTokPer slots a
// thread get their positions from a block scan; literals and match records go
// to the window's stage (a match's record at its first position, a bit in
// bm).  Then every position finds the last match start at or before it, and a
// position that the match covers takes its source: the history in the pages
// (or the marker / zero before the chunk), or a position of this window,
// followed by pointer jumping through the stage.  All positions of a window
// resolve in parallel, and a window without matches goes out as it is.
// Returns kOk, kBadDeflate (a distance beyond the window) or kPoolExhausted.
template <int LB>
__device__ __forceinline__ int32_t expand_tokens(CtaSmem<LB>* S, const PagePool& pool, uint32_t n,
                                                 uint32_t total_out, bool zero_window) {
  const uint32_t tid = threadIdx.x;
  const uint64_t o = S->c.o;
  const uint64_t base = o & ~(uint64_t)(kWin - 1);  // positions below are relative to this
  const uint32_t rel0 = (uint32_t)(o - base), rel_end = rel0 + total_out;
  uint32_t lo = rel0;          // next position to write
  uint32_t b0 = 0;             // first slot of the batch
  uint32_t bpos = rel0, bend;  // positions of the batch
  uint32_t pos[kTokPer], len[kTokPer], val[kTokPer], par = 0;
  for (uint32_t i = tid; i < kWin / 32; i += kCtaThreads) S->bm[i] = 0;
  if (tid == 0) {
    S->c.any_match = 0;
    S->c.carry_len = 0;
  }
  __syncthreads();
  auto load_batch = [&]() {
    const uint32_t i = b0 + kTokPer * tid;
    uint32_t sum = 0;
    uint32_t prev = 0;
    if (i < n) {
      const uint2 t = *reinterpret_cast<const uint2*>(S->tok + i);
      prev = i ? S->tok[i - 1] : 0u;
      val[0] = t.x & 0xFFFFu;
      val[1] = t.x >> 16;
      val[2] = t.y & 0xFFFFu;
      val[3] = t.y >> 16;
    } else {
      val[0] = val[1] = val[2] = val[3] = 0;
    }
#pragma unroll
    for (uint32_t k = 0; k < kTokPer; k++) {
      const uint32_t t = val[k];
      len[k] = i + k >= n ? 0u : (t & kTokMatch ? t & 0x1FFu : (prev & kTokMatch ? 0u : 1u));
      prev = t;
      pos[k] = sum;
      sum += len[k];
    }
    uint32_t a = sum, z = 0, ta, tz;
    cta_scan2(S, par, a, z, ta, tz);
    par ^= 1;
#pragma unroll
    for (uint32_t k = 0; k < kTokPer; k++) pos[k] += bpos + a;
    bend = bpos + ta;
  };
  load_batch();
  while (lo < rel_end) {
    const uint32_t wbase = lo & ~(kWin - 1), wend = wbase + kWin;
    if (!cta_page(S, pool, base + wbase)) return kPoolExhausted;
    for (;;) {
      // the batch's tokens that start in this window
#pragma unroll
      for (uint32_t k = 0; k < kTokPer; k++) {
        if (!len[k] || pos[k] < lo || pos[k] >= wend) continue;
        const uint32_t q = pos[k] - wbase;
        if (val[k] & kTokMatch) {
          const uint32_t d1 = S->tok[b0 + kTokPer * tid + k + 1];  // distance - 1
          S->stage[q] = len[k] << 16 | d1;
          atomicOr(&S->bm[q >> 5], 1u << (q & 31));
          S->c.any_match = 1;
          if ((uint64_t)d1 + 1 > base + pos[k] + kWindow) S->c.bad_dist = 1;
        } else {
          S->stage[q] = val[k];
        }
      }
      if (bend >= wend || b0 + kTokPer * kCtaThreads >= n) break;
      b0 += kTokPer * kCtaThreads;
      bpos = bend;
      load_batch();
    }
    __syncthreads();
    const uint32_t hi = min(wend, rel_end) - wbase, l0 = lo - wbase;
    uint16_t* page = pool.data + (size_t)S->c.page_cur * kPageEntries +
                     ((uint32_t)(base + wbase) & (kPageEntries - 1));
    const bool matches = S->c.any_match != 0 || S->c.carry_len != 0;
    if (matches) {
      const uint16_t* pprev = pool.data + (size_t)S->c.page_prev * kPageEntries;
      const uint16_t* pcur = pool.data + (size_t)S->c.page_cur * kPageEntries;
      const int32_t page_off = (int32_t)((uint32_t)(base + wbase) & (kPageEntries - 1));
      const int64_t wabs = (int64_t)(base + wbase);
      const int32_t c_ms = S->c.carry_ms;
      const uint32_t c_len = S->c.carry_len, c_dist = S->c.carry_dist;
      if (tid < kWin / 32) {
        int32_t m = -1;
        // a match is at most 258 long: nine words back
        for (int32_t w = (int32_t)tid - 1; w >= 0 && w + 9 >= (int32_t)tid; w--)
          if (S->bm[w]) {
            m = 32 * w + 31 - __clz(S->bm[w]);
            break;
          }
        S->lastm[tid] = m;
      }
      __syncthreads();
      // each position's new state: a value, or (bit 31) a reference into the window
      uint32_t st[kWinPer];
      uint32_t todo = 0;  // bit k: position k is covered by a match
#pragma unroll
      for (uint32_t k = 0; k < kWinPer; k++) {
        const uint32_t e = tid + kCtaThreads * k;
        st[k] = 0;
        if (e < l0 || e >= hi) continue;
        const uint32_t m = S->bm[e >> 5] & (0xFFFFFFFFu >> (31 - (e & 31)));
        int32_t ms = m ? (int32_t)((e & ~31u) + 31 - __clz(m)) : S->lastm[e >> 5];
        uint32_t ml, md;
        if (ms >= 0) {
          const uint32_t d = S->stage[ms];
          ml = d >> 16;
          md = (d & 0xFFFFu) + 1;
        } else {
          ms = c_ms;
          ml = c_len;
          md = c_dist;
        }
        const uint32_t jj = (uint32_t)((int32_t)e - ms);
        if (e + 1 == hi) {  // a match that goes on in the next window
          const bool more = jj < ml && (uint32_t)((int32_t)hi - ms) < ml;
          S->c.carry_ms = ms - (int32_t)kWin;
          S->c.carry_len = more ? ml : 0u;
          S->c.carry_dist = md;
        }
        if (jj >= ml) continue;
        todo |= 1u << k;
        // every entry of an overlapping match maps to one before the match
        const int32_t src = md < ml ? ms - (int32_t)md + (int32_t)(md == 1 ? 0u : jj % md)
                                    : (int32_t)e - (int32_t)md;
        if (src >= (int32_t)l0) {
          st[k] = 0x80000000u | (uint32_t)src;
        } else if (wabs + src >= 0) {
          const int32_t q = page_off + src;
          st[k] = q >= 0 ? pcur[q] : pprev[q + (int32_t)kPageEntries];
        } else {
          st[k] = zero_window ? 0u : (uint32_t)((int64_t)(kMarkerBase + kWindow) + wabs + src) & 0xFFFFu;
        }
      }
      __syncthreads();
#pragma unroll
      for (uint32_t k = 0; k < kWinPer; k++)
        if ((todo >> k) & 1) S->stage[tid + kCtaThreads * k] = st[k];
      // references: a position takes its source's value, or the source's own
      // reference (always further back), until none is left
      for (;;) {
        uint32_t left = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWinPer; k++) left |= st[k];
        if (!__syncthreads_or((int)(left >> 31))) break;
#pragma unroll
        for (uint32_t k = 0; k < kWinPer; k++)
          if (st[k] >> 31) {
            st[k] = *(volatile uint32_t*)&S->stage[st[k] & 0xFFFFu];
            *(volatile uint32_t*)&S->stage[tid + kCtaThreads * k] = st[k];
          }
      }
      if (tid < kWin / 32) S->bm[tid] = 0;
      if (tid == 0) S->c.any_match = 0;
      if (!zero_window) {
        uint32_t mk = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWinPer; k++)
          if (st[k] >= kMarkerBase) mk = tid + kCtaThreads * k + 1;
        mk = __reduce_max_sync(0xFFFFFFFFu, mk);
        if (mk && (tid & 31) == 0) atomicMax(&S->c.mark_max, mk);
      }
    }
    // out to the page, two entries per store
#pragma unroll
    for (uint32_t k = 0; k < kWinPer / 2; k++) {
      const uint32_t e = 2 * (tid + kCtaThreads * k);
      if (e + 1 < l0 || e >= hi) continue;
      const uint2 v = *reinterpret_cast<const uint2*>(&S->stage[e]);
      if (e >= l0 && e + 1 < hi) {
        *reinterpret_cast<uint32_t*>(page + e) = v.x | v.y << 16;
      } else if (e >= l0) {
        page[e] = (uint16_t)v.x;
      } else {
        page[e + 1] = (uint16_t)v.y;
      }
    }
    __syncthreads();
    if (S->c.bad_dist) return kBadDeflate;
    if (matches && !zero_window && tid == 0 && S->c.mark_max) {
      S->c.marker_end = base + wbase + S->c.mark_max;
      S->c.mark_max = 0;
    }
    lo = wbase + hi;
    if (bend <= wend && lo < rel_end) {
      b0 += kTokPer * kCtaThreads;
      bpos = bend;
      load_batch();
    }
  }
  return kOk;
}

// The body of one Huffman-coded block, tables in place.  On return (after a
// barrier) S->c holds the new position and entry count, status, synced (at
// the successor's sync start) or passed (went by the successor's start).
template <int LB>
__device__ __forceinline__ void cta_block(const uint8_t* __restrict__ in, CtaSmem<LB>* S,
                                          const PagePool& pool, bool zero_window) {
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(in);
  const uint32_t tid = threadIdx.x;
  uint32_t rcap = kRangeMax;
  for (;;) {
    // every thread computes the round's geometry from the shared state
    const uint64_t pos = S->c.pos, limit = S->c.limit_words, trunc = S->c.trunc_words;
    const uint64_t target = S->c.sync_target;
    const uint64_t w0 = pos >> 5;
    if (target == pos || w0 + 4 > limit) {
      __syncthreads();
      if (tid == 0) {
        if (target == pos) S->c.synced = 1;
        else S->c.status = w0 + 4 > trunc ? kTruncated : kOvershoot;
      }
      break;
    }
    uint64_t end = (limit - 3) * 32;  // symbols start below this
    if (target != kNoStop && target > pos && target < end) end = target;
    const uint64_t likely = S->c.stop_lo > pos && S->c.stop_lo < end ? S->c.stop_lo : end;
    const uint64_t want = ((likely - pos) / kCtaThreads + 32) & ~31ull;
    const uint32_t r = (uint32_t)max((uint64_t)kRangeMin, min(want, (uint64_t)rcap));
    const uint32_t p0 = (uint32_t)(pos & 31);
    const uint64_t span = end - pos;
    const uint32_t pend = p0 + (uint32_t)min(span, (uint64_t)r * kCtaThreads);
    const uint32_t lanes = (pend - p0 + r - 1) / r;
    // stage the input words (zeros past the stream's end)
    const uint32_t nw = (pend >> 5) + 6;
    for (uint32_t j = tid; j < nw; j += kCtaThreads)
      S->in[in_at(j)] = w0 + j < trunc ? in32[w0 + j] : 0u;
    if (tid < 2) S->c.min_need[tid] = S->c.min_term[tid] = kNone;
    __syncthreads();
    // 1. from the guessed starts
    const bool active = tid < lanes;
    const uint32_t e = min(p0 + (tid + 1) * r, pend);
    uint32_t start = p0 + tid * r;
    RangeOut ro{};
    if (active) {
      walk_range<LB, false>(S, start, e, tid > 0, ro, nullptr);
      S->end[tid] = ro.end;
    }
    // 2. from the end of the range before, until nothing moves
    uint32_t last = kNone;  // range that holds the end of the block (kNone: not in this round)
    for (uint32_t it = 0;; it ^= 1) {
      __syncthreads();
      const uint32_t s1 = active && tid ? S->end[tid - 1] : start;
      const bool need = active && s1 != start;
      const uint32_t mn = __reduce_min_sync(0xFFFFFFFFu, need ? tid : kNone);
      const uint32_t mt = __reduce_min_sync(0xFFFFFFFFu, active && ro.term ? tid : kNone);
      if ((tid & 31) == 0) {
        if (mn != kNone) atomicMin(&S->c.min_need[it], mn);
        if (mt != kNone) atomicMin(&S->c.min_term[it], mt);
      }
      __syncthreads();
      const uint32_t first_need = S->c.min_need[it];
      last = S->c.min_term[it];
      if (first_need == kNone || last < first_need) break;
      if (tid == 0) S->c.min_need[it ^ 1] = S->c.min_term[it ^ 1] = kNone;
      if (need) {
        start = s1;
        const uint32_t old = ro.end;
        walk_range<LB, false>(S, start, e, false, ro, nullptr);
        if (ro.term) ro.end = old;  // unknown past the stop: keep the guess
        S->end[tid] = ro.end;
      }
    }
    // 3. places in the token list; ranges beyond its capacity wait for the next round
    const uint32_t used = last != kNone ? last + 1 : lanes;
    const bool in_use = tid < used;
    uint32_t slots = in_use ? ro.slots : 0u, outs = in_use ? ro.outs : 0u, ts, to;
    const uint32_t my_slots = slots;
    cta_scan2(S, 0, slots, outs, ts, to);
    if (ts > kTokCap) {
      const uint32_t fit = (uint32_t)__syncthreads_count(in_use && slots + my_slots <= kTokCap);
      if (tid == fit) {
        S->c.round_slots = slots;
        S->c.round_out = outs;
        S->c.round_pos = start;  // = the end of range fit - 1
      }
      if (tid == 0) {
        S->c.round_lanes = fit;
        S->c.round_kind = kTermNone;
      }
      // shorter ranges from here on: about nine tenths of the list
      rcap = max(kRangeMin, min(rcap, (uint32_t)((uint64_t)r * kTokCap / ts * 9 / 10)) & ~31u);
    } else if (tid == used - 1) {
      S->c.round_slots = ts;
      S->c.round_out = to;
      S->c.round_lanes = used;
      S->c.round_kind = ro.term;
      S->c.round_pos = ro.term ? ro.term_pos : ro.end;
    }
    __syncthreads();
    const uint32_t n_lanes = S->c.round_lanes, n_slots = S->c.round_slots, n_out = S->c.round_out;
    const uint32_t kind = S->c.round_kind;
    const uint64_t new_pos = w0 * 32 + S->c.round_pos;
    if (kind == kTermBad) {
      __syncthreads();
      if (tid == 0) S->c.status = kBadDeflate;
      break;
    }
    if (tid < n_lanes) {
      RangeOut rw;
      walk_range<LB, true>(S, start, e, false, rw, S->tok + slots);
    }
    __syncthreads();
    // 4. expansion
    if (n_out) {
      const int32_t st = expand_tokens<LB>(S, pool, n_slots, n_out, zero_window);
      if (st != kOk) {
        __syncthreads();
        if (tid == 0) S->c.status = st;
        break;
      }
    }
    const bool passed = S->c.passed_bit < new_pos;
    __syncthreads();
    if (tid == 0) {
      S->c.pos = new_pos;
      S->c.o += n_out;
      if (kind == kTermNone && passed && new_pos != target) S->c.passed = 1;
    }
    __syncthreads();
    if (kind == kTermEob || S->c.passed) break;
  }
  __syncthreads();
}

// A stored block's bytes to the chunk's pages, four entries per thread.
template <int LB>
__device__ __forceinline__ void cta_stored(const uint8_t* __restrict__ in, CtaSmem<LB>* S,
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
    for (uint32_t g = (q & ~3u) + 4 * threadIdx.x; g < q + n; g += 4 * kCtaThreads) {
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
  __syncthreads();
  if (threadIdx.x == 0) {
    S->c.pos = byte * 8;
    S->c.o = o;
    if (!ok) S->c.status = kPoolExhausted;
  }
  __syncthreads();
}

// what the chunk does next
enum : int32_t {
  kActDone = 0,     // the chunk is finished (status)
  kActResume,       // the same block goes on, tables in place
  kActHeader,       // a block header at pos
  kActTable,        // a sync start: read the header at table_bit, then go on at pos
  kActFixed,        // a sync start in a fixed block
  kActStored,       // copy stored_len bytes at pos
  kActBlock,        // code lengths are read: build the tables, decode the block
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

// One warp: the boundary's decision and the header it leads to.
template <int LB>
__device__ __noinline__ void cta_header(const uint8_t* __restrict__ in, const ChunkDesc* descs,
                                        CtaSmem<LB>* S, const PagePool& pool, bool sync, int lane) {
  CtaCtl& c = S->c;
  int32_t act = kActDone;
  if (lane == 0) act = cta_boundary(c, descs, pool);
  act = __shfl_sync(0xFFFFFFFFu, act, 0);
  __syncwarp();
  int32_t status = kOk;
  if (act == kActHeader || act == kActTable) {
    BitReader br;
    br.in32 = reinterpret_cast<const uint32_t*>(in);
    br.limit_words = c.limit_words;
    const uint64_t start = act == kActTable ? c.table_bit : c.pos;
    br.load_windows((start >> 5) & ~31ull, lane);
    br.seek(start, lane);
    br.refill(lane);
    const uint32_t hdr = (uint32_t)br.bb & 7;
    br.consume(3);
    const uint32_t btype = hdr >> 1;
    uint64_t pos = c.pos;
    int nlen = 0, ndist = 0;
    uint32_t stored = 0;
    if (btype == 3 || (btype == 0 && act == kActTable)) {
      status = kBadDeflate;
    } else if (btype == 0) {
      // stored block: byte-align, LEN/NLEN
      br.consume(br.bc & 7);
      br.refill(lane);
      stored = (uint32_t)br.bb & 0xFFFF;
      const uint32_t nln = (uint32_t)(br.bb >> 16) & 0xFFFF;
      br.consume(32);
      const uint64_t byte = br.pos() >> 3;
      pos = byte * 8;
      if (byte > c.in_end) status = kTruncated;
      else if (stored != (~nln & 0xFFFFu)) status = kBadDeflate;
      else if (byte + stored > c.in_end) status = kTruncated;
    } else if (btype == 2 || !c.fixed_tables) {
      status = read_lens(br, btype, &S->h, c.trunc_words, lane, nlen, ndist);
      if (act == kActHeader) pos = br.pos();
    } else if (act == kActHeader) {
      pos = br.pos();
    }
    __syncwarp();
    if (lane == 0) {
      c.bfinal = hdr & 1;
      c.btype = btype;
      c.pos = pos;
      c.nlen = (uint32_t)nlen;
      c.ndist = (uint32_t)ndist;
      c.stored_len = stored;
    }
    act = btype == 0 ? kActStored : kActBlock;
  } else if (act == kActFixed) {
    BitReader br{};
    int nlen = 0, ndist = 0;
    if (!c.fixed_tables) read_lens(br, 1, &S->h, 0, lane, nlen, ndist);
    if (lane == 0) {
      c.nlen = (uint32_t)nlen;
      c.ndist = (uint32_t)ndist;
    }
    act = kActBlock;
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
template <int LB>
__device__ __forceinline__ void cta_decode_chunk(const uint8_t* __restrict__ in, const ChunkDesc* descs,
                                                 ChunkResult* res, CtaSmem<LB>* S,
                                                 const PagePool& pool, bool sync) {
  const int tid = threadIdx.x;
  CtaCtl& c = S->c;
  const bool zero_window = (c.flags & kChunkMemberFirst) != 0;
  for (;;) {
    if (tid < 32) cta_header<LB>(in, descs, S, pool, sync, tid);
    __syncthreads();
    const int32_t act = c.act;
    if (act == kActDone) break;
    if (act == kActStored) {
      cta_stored<LB>(in, S, pool);
    } else {
      if (act == kActBlock && !(c.btype == 1 && c.fixed_tables)) {
        const bool ok = cta_build_tables<LB>(S);
        if (tid == 0) {
          c.fixed_tables = c.btype == 1;
          if (!ok) c.status = kBadDeflate;
        }
        __syncthreads();
        if (!ok) {
          if (tid == 0) c.fixed_tables = 0;
          break;
        }
      }
      cta_block<LB>(in, S, pool, zero_window);
    }
    if (c.status != kOk || c.synced) break;
    const bool passed = c.passed != 0, fin = c.bfinal != 0;
    __syncthreads();
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
  __syncthreads();
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
  __syncthreads();
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
  c.bad_dist = c.mark_max = 0;
  c.bfinal = c.btype = 0;
  cta_set_limit(c);
}

}  // namespace gzgpu
