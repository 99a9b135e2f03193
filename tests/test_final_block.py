"""A member's final block as a start of its own: near the end of a member the
finder also takes headers with BFINAL set.  Survivors of its filter then lie
two bits apart at the closest (bits 1, 0, 1, 0, ... do), which the list of a
screening pass has to hold."""
import zlib

import numpy as np
import pytest

from gzippy_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, 8192])
def ctx(request):
    import gzippy_b200 as G
    c = G.Context(chunk_bytes=request.param)
    yield c
    c.close()


@pytest.mark.parametrize("kind", range(4))
@pytest.mark.parametrize("size", [20000, 65536, 100001, 400000, 1 << 20])
def test_last_blocks(ctx, kind, size):
    plain = W.content(kind, 77 + size % 89, size).tobytes()
    for level in (1, 6, 9):
        comp = W.gzip_member(np.frombuffer(plain, np.uint8), level).tobytes()
        assert ctx.decompress(comp) == plain
        assert ctx.decompress(comp + comp) == plain + plain


def test_the_final_block_is_a_chunk(ctx):
    plain = W.content(W.MARKOV, 5, 300000)
    assert ctx.decompress(W.gzip_member(plain, 6).tobytes()) == plain.tobytes()
    d, r = ctx.last_chunks()
    ends = r[(d["flags"] & 2 != 0) & (r["final_block"] != 0) & (r["status"] == 0)]
    assert (ends["n_blocks"] <= 1).any()


@pytest.mark.parametrize("fill", [0x55, 0xAA, 0x2D, 0x05, 0x00, 0xFF])
@pytest.mark.parametrize("n", [40, 5000, 70000])
def test_bytes_after_the_member(ctx, fill, n):
    """The last partitions hold one pattern, where up to every second bit
    passes the filter."""
    plain = W.content(W.MARKOV, 6, 150000)
    comp = W.gzip_member(plain, 6).tobytes()
    assert ctx.decompress(comp + bytes([fill]) * n) == plain.tobytes()


def test_patterns_inside_coded_data(ctx):
    """Eight-bit codes spell the same patterns in the data itself: raw DEFLATE,
    fixed code, so that the partitions are searched."""
    plain = bytes(range(144)) * 900
    co = zlib.compressobj(6, zlib.DEFLATED, -15, 8, zlib.Z_HUFFMAN_ONLY)
    comp = co.compress(plain) + co.flush()
    assert ctx.inflate_raw(comp) == plain


@pytest.mark.parametrize("bits", [1000, 1024, 1056, 8191, 16384, 70000, 196608])
def test_search_of_few_and_of_many_ranges(ctx, bits):
    """A small search is cut into shorter segments, one warp each: the first
    start of a range is the same in both."""
    comp = W.gzip_member(W.content(W.MARKOV, 8, 400000), 6)
    total = comp.size * 8
    for lo in range(100, total - bits, max(bits, 100003)):
        alone = ctx.debug_find(comp, [(lo, lo + bits)])
        assert ctx.debug_find(comp, [(lo, lo + bits)] * 600) == alone * 600
