"""A stream cut off inside a dynamic block's header: its status follows from
where the reading of the code lengths stops.  A symbol more than 64 bits past the
input is out of reach, so the stream is cut off (TRUNCATED); one before that which
is no code, or repeats past the last length, makes it invalid (BAD_DEFLATE).
Expected: a serial reading of the same bytes (RFC 1951 3.2.7), including the
readable ones after the input that the device entry points are given."""
import ctypes

import numpy as np
import pytest

from gzippy_b200 import workloads as W

pytestmark = pytest.mark.gpu

ORDER = [16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15]


def _expected(data, n, at):
    """Status of the member of n bytes whose dynamic header starts at byte `at`
    of data, or None when the header reads through."""
    import gzippy_b200 as G
    bits = np.unpackbits(data, bitorder="little")

    def get(p, k):
        return int(sum(int(bits[p + i]) << i for i in range(k)))

    p = at * 8
    assert get(p, 3) >> 1 == 2
    total, ncl = 258 + get(p + 3, 5) + get(p + 8, 5), 4 + get(p + 13, 4)
    lens = [0] * 19
    for i in range(ncl):
        lens[ORDER[i]] = get(p + 17 + 3 * i, 3)
    codes, code = {}, 0
    for ln in range(1, 8):
        code <<= 1
        for s in range(19):
            if lens[s] == ln:
                codes[ln, code] = s
                code += 1
    p += 17 + 3 * ncl
    limit = ((n * 8 + 31) // 32 + 5) * 32
    i = 0
    while i < total:
        if p + 96 >= limit:
            return G.TRUNCATED
        code = 0
        for ln in range(1, 8):
            code = code << 1 | get(p + ln - 1, 1)
            if (ln, code) in codes:
                break
        else:
            return G.BAD_DEFLATE
        s, p = codes[ln, code], p + ln
        k = {16: 2, 17: 3, 18: 7}.get(s, 0)
        rep = 1 if s < 16 else get(p, k) + (11 if s == 18 else 3)
        p += k
        if (s == 16 and i == 0) or i + rep > total:
            return G.BAD_DEFLATE
        i += rep
    return None


@pytest.mark.parametrize("fill", [0x00, 0x77, 0x5A, 0xFF])
@pytest.mark.parametrize("size,seed", [(3000, 5), (700, 14), (900, 1)])
def test_cut_inside_the_code_lengths(size, seed, fill):
    import torch

    import gzippy_b200 as G
    comp = W.gzip_member(W.content(W.MARKOV, seed, size), 9)
    cx = G.Context()
    seen = set()
    try:
        d_in = torch.empty(8192, dtype=torch.uint8, device="cuda")
        d_out = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
        for cut in range(10 + 3 + 7, 120):
            data = np.full(8192, fill, np.uint8)
            data[:cut] = comp[:cut]
            want = _expected(data, cut, 10)
            if want is None:
                continue
            seen.add(want)
            d_in.copy_(torch.from_numpy(data))
            torch.cuda.synchronize()
            got = ctypes.c_size_t(0)
            rc = cx._lib.gzgpu_decompress_device(cx._h, d_in.data_ptr(), cut, d_out.data_ptr(), 1 << 20,
                                                 ctypes.byref(got))
            assert rc == want, cut
            rc = cx._lib.gzgpu_decompress_device_noalloc(d_in.data_ptr(), cut, d_out.data_ptr(), 1 << 20,
                                                         ctypes.byref(got), None)
            assert rc == want, cut
        assert seen
    finally:
        cx.close()
