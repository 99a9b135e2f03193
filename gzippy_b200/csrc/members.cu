// members.cu -- gzip member location on the device.
//
// stream_info: per stream, the magic check (non-gzip -> kNotGzip,
//   src/lib.rs:50-52) and the first member's header length (RFC 1952,
//   gzip_format.rs read_header :47-133).
// member_scan_kernel: every byte position of every stream is tested like
//   scan_member_boundaries_fast (src/decompress/bgzf.rs:2090-2230): bytes
//   1f 8b 08, FLG & 0xE0 == 0, pos >= 4, the preceding ISIZE in (0, 1 GiB],
//   pos past the first header and pos + 10 < stream length; plus the header
//   plausibility of is_likely_multi_member (src/decompress/format.rs:92-125:
//   MTIME, XFL, OS), which removes nearly every false hit in compressed data.
//   A real member that fails it is still found by the host chain walk.
//   Each hit's header is parsed (parse_gzip_header :2047) for its deflate
//   start.
#include <cstdint>

#include "barrier.cuh"
#include "common.cuh"
#include "members.cuh"

namespace gzgpu {

// bit 7 of each byte of the result is set exactly where w's byte is zero
__device__ __forceinline__ uint32_t zero_bytes(uint32_t w) {
  const uint32_t t = (w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu;
  return ~(t | w | 0x7F7F7F7Fu);
}

// the first zero byte of in from o on, lim when there is none before it
struct ThreadFindZero {
  __device__ uint64_t operator()(const uint8_t* in, uint64_t o, uint64_t lim) const {
    while (o < lim && in[o]) o++;
    return o;
  }
};
// The same by a whole warp, 2 KiB a step (in: 16-byte aligned): a comment of
// 60 KB is 60,000 loads one after another for a thread, 3 ms and more where every
// CTA reads it (a 22 MB stream's scan: 14 ms).
struct WarpFindZero {
  uint32_t lane;
  __device__ uint64_t operator()(const uint8_t* in, uint64_t o, uint64_t lim) const {
    for (uint64_t base = o & ~15ull; base < lim; base += 2048) {
      uint4 v[4];
#pragma unroll
      for (uint32_t j = 0; j < 4; j++) {
        const uint64_t a = base + 512 * j + 16 * lane;
        v[j] = a < lim ? *reinterpret_cast<const uint4*>(in + a) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (uint32_t j = 0; j < 4; j++) {
        const uint64_t a = base + 512 * j + 16 * lane;
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        uint32_t first = 16;
#pragma unroll
        for (int k = 3; k >= 0; k--) {
          uint32_t z = zero_bytes(w[k]);
          if (a + 4 * k < o) z = a + 4 * k + 4 <= o ? 0u : z & 0xFFFFFFFFu << (8 * (uint32_t)(o - a - 4 * k));
          if (z) first = 4 * k + ((__ffs(z) - 1) >> 3);
        }
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, first < 16);
        if (b) {
          const uint32_t src = __ffs(b) - 1;
          const uint64_t at = base + 512 * j + 16 * src + __shfl_sync(0xFFFFFFFFu, first, src);
          return at < lim ? at : lim;
        }
      }
    }
    return lim;
  }
};

// header length of the member at `p` (absolute), bounded by `end`;
// returns 0 on a malformed or truncated header.
template <typename FindZero>
__device__ uint64_t parse_header(const uint8_t* in, uint64_t p, uint64_t end, FindZero find_zero) {
  if (end < p + 10) return 0;
  if (in[p] != 0x1f || in[p + 1] != 0x8b || in[p + 2] != 8) return 0;
  uint8_t flg = in[p + 3];
  if (flg & 0xE0) return 0;
  uint64_t o = p + 10;
  if (flg & 4) {
    if (o + 2 > end) return 0;
    uint64_t xlen = in[o] | (in[o + 1] << 8);
    o += 2 + xlen;
    if (o > end) return 0;
  }
  for (int f = 8; f <= 16; f <<= 1) {
    if (flg & f) {
      const uint64_t lim = min(end, o + 65536);  // bounded walk
      o = find_zero(in, o, lim);
      if (o >= lim) return 0;
      o++;
    }
  }
  if (flg & 2) {
    o += 2;
    if (o > end) return 0;
  }
  return o - p;
}

// by one warp; not inlined, so that the scan keeps its registers
__device__ __noinline__ StreamInfo stream_info(const uint8_t* __restrict__ in, uint64_t p, uint64_t len, uint32_t lane) {
  StreamInfo si{};
  if (len < 2 || in[p] != 0x1f || in[p + 1] != 0x8b) {
    si.status = kNotGzip;
  } else {
    uint64_t h = parse_header(in, p, p + len, WarpFindZero{lane});
    if (h == 0) {
      si.status = (len < 10 || in[p + 2] == 8) ? kTruncated : kBadHeader;
      if (len >= 10 && in[p + 2] == 8 && (in[p + 3] & 0xE0)) si.status = kBadHeader;
    } else {
      si.status = kOk;
      si.header_len = (uint32_t)h;
    }
  }
  si.first_btype = 4;
  if (si.status == kOk && si.header_len < len) si.first_btype = (in[p + si.header_len] >> 1) & 3;
  if (len >= 4) {
    const uint8_t* t = in + p + len - 4;
    si.last_isize = t[0] | (t[1] << 8) | ((uint32_t)t[2] << 16) | ((uint32_t)t[3] << 24);
  }
  return si;
}

// grid-stride over scan units (stream, byte range); the first warp of every CTA
// reads the stream's first header for itself (a kernel for that alone would be
// one more wait) and the first unit's writes it down; each thread screens 16
// aligned bytes at a time for the 0x1f of the magic with word operations and
// tests only the positions that have one
constexpr int kScanThreads = 512;
__global__ void __launch_bounds__(kScanThreads, 4)
    member_scan_kernel(const uint8_t* __restrict__ in, const ScanUnit* __restrict__ units, uint32_t n_units,
                       const uint64_t* __restrict__ s_off, const uint64_t* __restrict__ s_len,
                       StreamInfo* info, MemberCand* cands, uint32_t* n_cands, uint32_t cap) {
  __shared__ StreamInfo s_info;
  uint32_t known = 0xFFFFFFFFu;  // the stream s_info is of
  for (uint32_t u = blockIdx.x; u < n_units; u += gridDim.x) {
    const ScanUnit su = units[u];
    const uint64_t base = s_off[su.stream], len = s_len[su.stream];
    cta_sync();  // the unit before has read s_info
    if (threadIdx.x < 32) {
      const StreamInfo si = su.stream != known ? stream_info(in, base, len, threadIdx.x) : s_info;
      __syncwarp();
      if (threadIdx.x == 0) {
        s_info = si;
        if (su.begin == 0) info[su.stream] = si;
      }
    }
    cta_sync();
    known = su.stream;
    const StreamInfo si = s_info;
    if (si.status != kOk) continue;
    const uint64_t lo = su.begin > (uint64_t)si.header_len + 1 ? su.begin : si.header_len + 1;
    for (uint64_t a = ((base + lo) & ~15ull) + 16 * (uint64_t)threadIdx.x; a < base + su.end;
         a += 16 * (uint64_t)blockDim.x) {
      const uint4 v = *reinterpret_cast<const uint4*>(in + a);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        uint32_t m = zero_bytes(w[k] ^ 0x1F1F1F1Fu);
        while (m) {
          const int j = (__ffs(m) - 1) >> 3;
          m &= m - 1;
          const uint64_t pos = a + 4 * k + j - base;
          if (pos < lo || pos >= su.end) continue;
          if (pos + 10 >= len || pos < 4) continue;
          const uint8_t* q = in + base + pos;
          if (q[0] != 0x1f || q[1] != 0x8b || q[2] != 8 || (q[3] & 0xE0)) continue;
          const uint32_t isz =
              q[-4] | (q[-3] << 8) | ((uint32_t)q[-2] << 16) | ((uint32_t)q[-1] << 24);
          if (isz == 0 || isz > (1u << 30)) continue;
          // header plausibility of is_likely_multi_member (format.rs:92-125):
          // MTIME 0 or <= 4102444800, XFL in {0, 2, 4}, OS <= 13 or 255
          const uint32_t mtime =
              q[4] | (q[5] << 8) | ((uint32_t)q[6] << 16) | ((uint32_t)q[7] << 24);
          if (mtime > 4102444800u) continue;
          if (q[8] != 0 && q[8] != 2 && q[8] != 4) continue;
          if (q[9] > 13 && q[9] != 255) continue;
          const uint32_t kk = atomicAdd(n_cands, 1u);
          if (kk < cap) {
            MemberCand c;
            c.stream = su.stream;
            c.pos = pos;
            c.header_len = (uint32_t)parse_header(in, base + pos, base + len, ThreadFindZero{});
            c.prev_isize = isz;
            cands[kk] = c;
          }
        }
      }
    }
  }
}

cudaError_t launch_member_scan(const uint8_t* in, const ScanUnit* units, uint32_t n_units,
                               const uint64_t* s_off, const uint64_t* s_len, StreamInfo* info,
                               MemberCand* cands, uint32_t* n_cands, uint32_t cap, int sms,
                               cudaStream_t stream) {
  if (!n_units) return cudaSuccess;
  uint32_t grid = n_units < (uint32_t)(sms * 16) ? n_units : (uint32_t)(sms * 16);
  member_scan_kernel<<<grid, kScanThreads, 0, stream>>>(in, units, n_units, s_off, s_len, info, cands,
                                                n_cands, cap);
  return cudaGetLastError();
}

}  // namespace gzgpu
