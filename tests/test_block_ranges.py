"""The page-history block decoder where its pieces meet.

A Huffman block is decoded as bit ranges, one per thread, joined where they
resynchronise, and its tokens are expanded in windows of 2048 entries.  These
inputs put block ends, window and page edges, token-list overflow, codes that
hardly resynchronise and long reference chains in its way.  Integer work:
every chunk's entries, end bit and marker end equal the oracle's, exactly."""
import zlib

import numpy as np
import pytest

from gzippy_b200 import workloads as W
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

HUFF = zlib.Z_HUFFMAN_ONLY


def _rng():
    return np.random.default_rng(77)


def _gz(p, level=6, strategy=zlib.Z_DEFAULT_STRATEGY):
    o = zlib.compressobj(level, zlib.DEFLATED, 31, 8, strategy)
    return np.frombuffer(o.compress(np.ascontiguousarray(p, np.uint8).tobytes()) + o.flush(), np.uint8)


def _runs(lo, hi, n):
    r = _rng()
    return np.repeat(r.integers(0, 256, n), r.integers(lo, hi, n)).astype(np.uint8)


CASES = {
    # window (2048) and page (65536) edges, by output size
    **{f"text_{n}": lambda n=n: _gz(W.content(W.MARKOV, n, n))
       for n in (1, 2, 2047, 2048, 2049, 4097, 65535, 65536, 65537, 131073)},
    # one match reaching over many windows; 2 bits per 258 bytes
    "zeros": lambda: _gz(np.zeros(3_000_000)),
    # 1-bit codes: more tokens in a round than its list holds
    "bits_huffman": lambda: _gz(_rng().integers(0, 2, 600_000), 6, HUFF),
    "geometric_huffman": lambda: _gz(np.minimum(_rng().geometric(0.5, 400_000), 255), 6, HUFF),
    # codes of nearly one length hardly resynchronise
    "six_bit_huffman": lambda: _gz(_rng().integers(0, 64, 300_000) + 32, 6, HUFF),
    "bytes_huffman": lambda: _gz(np.minimum(_rng().normal(128, 60, 300_000).clip(0, 255), 255), 6, HUFF),
    # long chains of references inside a window, overlapping and not
    "periodic": lambda: _gz(np.tile(_rng().integers(0, 256, 777), 3000)),
    "short_runs": lambda: _gz(_runs(1, 9, 80_000), 9),
    "long_runs": lambda: _gz(_runs(200, 700, 4_000), 9),
    "fixed_codes": lambda: W.gzip_member(W.content(W.MARKOV, 3, 500_000), 1),
}


@pytest.fixture(scope="module")
def ctx():
    import gzippy_b200 as G
    c = G.Context()
    yield c
    c.close()


@pytest.mark.parametrize("name", list(CASES))
def test_block_ranges_match_oracle(ctx, name):
    c = CASES[name]()
    _, hl = O.gzip_header_len(c)
    nbits, none = c.size * 8, 2**64 - 1
    starts, step = [], 24 * 1024 * 8
    for g in range(hl * 8 + step, nbits - 1000, step):
        first, seek = O.find_blocks(c, g, min(g + step, nbits), cap=4)
        if first.size:
            starts.append((int(first[0]), int(seek[0])))
    # the member's first chunk (zero window) and chunks with markers
    chunks = [(hl * 8, starts[0][0] if starts else none, True)]
    for k, (lo, hi) in enumerate(starts):
        chunks.append((hi, starts[k + 1][0] if k + 1 < len(starts) else none, False))
    cap = 4 << 20
    res, ent = ctx.debug_decode(c, chunks, cap)
    for i, (s, stop, mf) in enumerate(chunks):
        st, r, e = O.inflate_chunk(c, s, stop, markers=not mf, cap=cap)
        assert int(res[i, 4]) == st, i
        if st != O.OK:
            continue
        assert [int(x) for x in res[i, :4]] == [r.end_bit, r.out_len, r.marker_end, r.n_blocks], i
        assert np.array_equal(ent[i, :r.out_len], e), i
