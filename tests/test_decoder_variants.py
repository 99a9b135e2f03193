"""The page-history decoder's variants: CTAs of 256 threads (jobs of over two chunks
per SM, three or four CTAs per SM) and of 1,024, tables of 10 to 12 bits.  Integer
work: bytes and entries equal the oracle's and zlib's exactly."""
import zlib

import numpy as np
import pytest

from gzippy_b200 import workloads as W
from oracle import pyoracle as O
from test_block_ranges import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk_bytes", [4096, 65536])  # over, and up to, two chunks per SM
@pytest.mark.parametrize("ctas_per_sm", [3, 4])
@pytest.mark.parametrize("lut_bits", [10, 11, 12])
def test_streams(lut_bits, ctas_per_sm, chunk_bytes):
    import gzippy_b200 as G
    parts = [W.content(k % 4, 30 + k, 1200001) for k in range(8)]
    parts.append(np.random.default_rng(3).geometric(0.02, 400000).clip(0, 255).astype(np.uint8))  # long codes
    plain = np.concatenate(parts)
    cx = G.Context(chunk_bytes=chunk_bytes, lut_bits=lut_bits, ctas_per_sm=ctas_per_sm)
    try:
        for level in (1, 6, 9):
            assert cx.decompress(W.gzip_member(plain, level)) == plain.tobytes()
            n = int((cx.last_chunks()[0]["flags"] & 2 != 0).sum())
            if level == 9:
                assert (n > 2 * 148) == (chunk_bytes == 4096)
    finally:
        cx.close()


@pytest.mark.parametrize("name", ["text_1", "text_2047", "text_2048", "text_2049", "text_4097", "text_65535",
                                  "text_65536", "text_65537", "text_131073", "bits_huffman", "geometric_huffman",
                                  "six_bit_huffman", "periodic", "short_runs", "fixed_codes"])
def test_blocks_in_narrow_ctas(name):
    """test_block_ranges decodes its few chunks with 1,024 threads each; here the
    first and a middle one are so many that they get 256."""
    import gzippy_b200 as G
    c = CASES[name]()
    _, hl = O.gzip_header_len(c)
    nbits, none = c.size * 8, 2**64 - 1
    chunks = [(hl * 8, none, True)]
    first, seek = O.find_blocks(c, hl * 8 + 8 * 24 * 1024, nbits, cap=4) if nbits > 8 * 30000 else ((), ())
    if len(first):
        chunks.append((int(seek[0]), none, False))
    cap = 200000
    many = chunks * 150 if len(chunks) == 2 else chunks * 300
    cx = G.Context()
    try:
        res, ent = cx.debug_decode(c, many, cap)
        for i, (s, stop, mf) in enumerate(chunks):
            st, r, e = O.inflate_chunk(c, s, stop, markers=not mf, cap=4 << 20)
            for k in (i, len(many) - len(chunks) + i):
                assert int(res[k, 4]) == st
                if st != O.OK:
                    continue
                assert [int(x) for x in res[k, :4]] == [r.end_bit, r.out_len, r.marker_end, r.n_blocks]
                m = min(cap, r.out_len)
                assert np.array_equal(ent[k, :m], e[:m])
    finally:
        cx.close()


def test_fixed_codes_that_pass_the_header_filter():
    """Literals whose fixed codes spell 1, 0, 1, 0, ...: near a member's end every
    second bit of them passes the filter for the header of a final block."""
    import gzippy_b200 as G
    for lit, bits in ((0x7A, 0xAA), (0x25, 0x55)):
        n = 60000
        body = np.unpackbits(np.full(n, bits, np.uint8))  # a code's first bit is its most significant
        b = np.concatenate([[1, 1, 0], body, np.zeros(7, np.uint8)]).astype(np.uint8)  # BFINAL, BTYPE 01, end of block
        raw = np.packbits(b, bitorder="little").tobytes()
        assert raw[0] >> 1 & 3 == 1 and zlib.decompress(raw, -15) == bytes([lit]) * n
        for chunk_bytes in (0, 2048):
            cx = G.Context(chunk_bytes=chunk_bytes)
            try:
                assert cx.inflate_raw(raw) == bytes([lit]) * n
            finally:
                cx.close()
