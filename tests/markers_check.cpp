// CPU check of the marker walk (gzippy_b200/csrc/markers.cuh) against a 64-bit
// model, over placed chunks of made-up output.
//
// Every byte of a member is a function of its offset: a period of bytes, or 0
// before the member.  An entry of a chunk is the byte itself where the chunk is
// a literal one, else the marker of the place one or more periods back that lies
// before the chunk, as a decoder that starts there gives it.  Pages hold nothing:
// an entry is computed from its page's chunk and number when it is asked for, so
// members of any length can be walked; a page that no chunk names, and an entry
// past a chunk's end, count as failures.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../gzippy_b200/csrc/markers.cuh"

using namespace gzgpu;

namespace {

int failures = 0, checked = 0;

struct Member {
  std::vector<PlacedChunk> placed;
  std::vector<uint64_t> len;
  std::vector<bool> literal;
  uint64_t moff = 0;
  uint32_t period = 1;

  uint32_t byte(uint64_t x) const { return (uint32_t)((x - moff) % period * 37 + 11) & 0xFF; }

  void add(uint64_t n, bool lit) {
    const uint64_t off = placed.empty() ? moff : placed.back().out_off + len.back();
    const uint32_t k = (uint32_t)placed.size();
    const uint32_t last = n ? (uint32_t)((n - 1) / kPageEntries) : 0u;
    placed.push_back(PlacedChunk{off, moff, k, n ? 2 * k + 1 : kNoPage, last ? 2 * k : kNoPage, last});
    len.push_back(n);
    literal.push_back(lit);
  }
  uint32_t entry(uint32_t k, uint64_t q) const {
    const uint64_t off = placed[k].out_off;
    if (literal[k]) return byte(off + q);
    return 65536 - (period - (uint32_t)(q % period));  // the same place of the period before the chunk
  }
  uint32_t at_page(uint32_t page, uint32_t i) const {
    const uint32_t k = page / 2;
    if (page == kNoPage || k >= placed.size()) {
      failures++;
      return 0;
    }
    const uint64_t q = ((uint64_t)placed[k].last_seq - (page % 2 ? 0 : 1)) * kPageEntries + i;
    if (q >= len[k]) {
      failures++;
      return 0;
    }
    return entry(k, q);
  }
  // the byte that marker v of chunk k names
  void check(uint32_t k, uint32_t v) {
    const uint64_t off = placed[k].out_off;
    NearChunk near[kNear];
    for (uint32_t i = 0; i < kNear && i < k; i++) near[i] = near_chunk(placed[k - 1 - i]);
    const uint32_t got = follow_marker(placed.data(), near, k, off, moff, v,
                                       [&](uint32_t page, uint32_t i) { return at_page(page, i); });
    const uint64_t dist = 65536 - v;
    const uint32_t want = dist > off - moff ? 0u : byte(off - dist);
    checked++;
    if (got != want && failures++ < 20)
      printf("period %u chunk %u at %llu marker %u: %u, not %u\n", period, k, (unsigned long long)off, v, got, want);
  }
  void check_all() {
    for (uint32_t k = 0; k < placed.size(); k++)
      for (uint32_t v : {32768u, 32769u, 40000u, 65535u - period, 65536u - period, 65534u, 65535u}) check(k, v);
  }
};

}  // namespace

int main() {
  // over 4 GiB of one repetition: every chunk but the first is all markers
  for (uint32_t period : {1u, 2u, 3u, 100u, 1024u, 32768u}) {
    Member m;
    m.period = period;
    m.moff = 12345;
    m.add(70000, true);
    while (m.placed.back().out_off < 5ull << 30) m.add(25000003, false);
    m.check_all();
  }
  // one chunk that alone gives over 4 GiB
  for (uint64_t n : {(4ull << 30) - 1, 4ull << 30, (4ull << 30) + 65537, (9ull << 30) + 3}) {
    for (bool lit : {true, false}) {
      Member m;
      m.period = 7;
      m.add(40000, true);
      m.add(n, lit);
      m.add(50000, false);
      m.add(100, false);
      m.check_all();
    }
  }
  // short and empty chunks, windows that reach before the member
  for (uint32_t period : {1u, 5u, 300u}) {
    Member m;
    m.period = period;
    m.moff = 999;
    m.add(period + 7, true);
    for (int i = 0; i < 300; i++) m.add((uint64_t)(i % 4 ? i % 7 : 0) * 1000, false);
    m.add(65536, false);
    m.add(65537, false);
    m.add(131072, false);
    m.add(1, false);
    m.check_all();
  }
  printf("%d checked, %d failures\n", checked, failures);
  return failures != 0;
}
