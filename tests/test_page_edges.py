"""Chunks that end exactly on a page (65,536 entries) in a block of about as
many token slots as the decoder's batches hold.

A match takes two slots, its length and its distance.  When the last batch of a
block holds only the distance, it has no output, and must not open a window or
take a page: the next chunk's references are looked up in the page that its
predecessor names as its last.  The blocks here have 1,023 to 1,026 and 4,095 to
4,098 slots (batches are 1,024 slots in CTAs of 256 threads, 4,096 in those of
1,024), end in a match and on 65,536 or 131,072 bytes, and the block after each
copies from its last 32 KiB.  Raw DEFLATE, which has no checksum to fail;
bytes are compared exactly."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEN_BASE = [3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 15, 17, 19, 23, 27, 31, 35, 43, 51, 59, 67, 83, 99, 115,
            131, 163, 195, 227, 258]
LEN_EXTRA = [0] * 8 + [1] * 4 + [2] * 4 + [3] * 4 + [4] * 4 + [5] * 4 + [0]


def _fixed_block(slots, size, seed):
    """A non-final fixed-code block (RFC 1951 3.2.6) of `slots` token slots and
    `size` bytes that ends in a match, then the empty stored block that fills up
    the last byte."""
    rng = np.random.default_rng(seed)
    n_match = size // 258 + 12
    lens = np.full(n_match, 258)
    over = int(lens.sum()) + slots - 2 * n_match - size
    for i in range(n_match):
        cut = min(over, 200)
        lens[i] -= cut
        over -= cut
    assert over == 0 and slots >= 2 * n_match
    bits = [0, 1, 0]  # BFINAL 0, BTYPE 01

    def code(value, n):
        bits.extend((value >> i) & 1 for i in range(n - 1, -1, -1))

    for lit in rng.integers(0, 144, slots - 2 * n_match):
        code(0x30 + int(lit), 8)
    for n in lens:
        k = 28 if n == 258 else max(i for i in range(28) if LEN_BASE[i] <= n)
        sym = 257 + k
        code(sym - 256, 7) if sym < 280 else code(0xC0 + sym - 280, 8)
        bits.extend(((int(n) - LEN_BASE[k]) >> i) & 1 for i in range(LEN_EXTRA[k]))
        code(9, 5)  # distance 25 to 32
        bits.extend((1, 0, 1))
    code(0, 7)
    bits.extend((0, 0, 0))
    bits.extend([0] * (-len(bits) % 8))
    return np.packbits(np.array(bits, np.uint8), bitorder="little").tobytes() + b"\x00\x00\xff\xff"


def _copying_block(window, size, seed, any_type=False):
    """A dynamic block of `size` bytes, pieces of the 32 KiB before it between
    bytes of its own, then an empty stored block."""
    rng = np.random.default_rng(seed)
    parts, n = [], 0
    while n < size:
        at = int(rng.integers(0, len(window) - 300))
        parts += [window[at:at + int(rng.integers(100, 259))],
                  rng.integers(0, 256, int(rng.integers(1, 9)), dtype=np.uint8).tobytes()]
        n += len(parts[-1]) + len(parts[-2])
    plain = b"".join(parts)[:size]
    c = zlib.compressobj(9, zlib.DEFLATED, -15, 9, zlib.Z_DEFAULT_STRATEGY, window)
    comp = c.compress(plain) + c.flush(zlib.Z_SYNC_FLUSH)
    assert any_type or comp[0] & 7 == 4  # dynamic
    return comp


def _stream(slots, size, units):
    d = zlib.decompressobj(-15)
    comp, window, plain = [], b"", []
    for u in range(units):
        # the second kind of block gives a whole page too, so that every chunk
        # (from one of those on: a fixed block is no start) ends on a page
        for part in (_fixed_block(slots, size, u % 7), None):
            if part is None:
                part = _copying_block(window, 65536, u)
            comp.append(part)
            plain.append(d.decompress(part))
            window = (window + plain[-1])[-32768:]
    comp.append(b"\x03\x00")  # an empty final block
    return b"".join(comp), b"".join(plain)


# (slots, size, units): over two chunks per SM run CTAs of 256 threads, up to
# that many CTAs of 1,024
@pytest.mark.parametrize("slots", [1023, 1024, 1025, 1026])
def test_one_slot_past_a_batch_narrow(slots):
    _check(slots, 65536, 420, narrow=True)


@pytest.mark.parametrize("size", [65536, 131072])
@pytest.mark.parametrize("slots", [4095, 4096, 4097, 4098])
def test_one_slot_past_a_batch_wide(slots, size):
    _check(slots, size, 12, narrow=False)


def test_one_slot_past_four_batches_narrow():
    _check(4097, 131072, 420, narrow=True)


def _check(slots, size, units, narrow):
    import gzippy_b200 as G
    comp, plain = _stream(slots, size, units)
    cx = G.Context(chunk_bytes=1024)  # (too short for the search of fixed blocks)
    try:
        got = cx.inflate_raw(comp)
        assert got == plain
        d, r = cx.last_chunks()
        valid = d["flags"] & 2 != 0
        assert (int(valid.sum()) > 2 * 148) == narrow
        used = r[valid & (r["status"] == 0)]
        assert (used["out_len"] % 65536 == 0).sum() >= units // 2  # chunks that end on a page
        # no page without an entry
        assert np.array_equal(used["n_pages"], -(-used["out_len"].astype(np.int64) // 65536))
    finally:
        cx.close()


@pytest.mark.parametrize("seed", range(4))
def test_chunks_of_every_length(seed):
    """Chunks shorter and longer than a window, a page and a resolve unit (512
    entries), whose last 32 KiB are resolved apart from the rest, each copying from
    what lies before it."""
    import gzippy_b200 as G
    rng = np.random.default_rng(seed)
    sizes = [511, 512, 513, 3000, 32255, 32256, 32767, 32768, 32769, 33279, 33280, 33281, 65535, 65536, 65537,
             98303, 98304, 98305, 131072, 200001]
    d = zlib.decompressobj(-15)
    comp, window, plain = [], rng.integers(0, 256, 32768, dtype=np.uint8).tobytes(), []
    comp.append(b"".join(b"\x00" + n.to_bytes(2, "little") + (n ^ 0xFFFF).to_bytes(2, "little") + window
                         for n in (32768,)))
    plain.append(d.decompress(comp[0]))
    for i in rng.permutation(np.tile(sizes, 12)):
        comp.append(_copying_block(window, int(i), int(rng.integers(1 << 30)), any_type=True))
        plain.append(d.decompress(comp[-1]))
        window = (window + plain[-1])[-32768:]
    comp.append(b"\x03\x00")
    raw, plain = b"".join(comp), b"".join(plain)
    for chunk_bytes in (1024, 4096, 0):
        cx = G.Context(chunk_bytes=chunk_bytes)
        try:
            assert cx.inflate_raw(raw) == plain
        finally:
            cx.close()


@pytest.mark.parametrize("period", [1, 2, 100, 5000, 32768])
def test_repetition_over_many_chunks(period):
    """Every chunk but the first is all markers, and chains lead back over all."""
    import gzippy_b200 as G
    rec = np.random.default_rng(period).integers(0, 256, period, dtype=np.uint8)
    plain = np.tile(rec, (48 << 20) // period + 1).tobytes()
    comp = zlib.compressobj(9 if period < 32768 else 6, zlib.DEFLATED, 31)
    comp = comp.compress(plain) + comp.flush()
    cx = G.Context(chunk_bytes=1024)
    try:
        assert cx.decompress(comp) == plain
        assert cx.stats().n_accepted > (8 if period > 1 else 2)
    finally:
        cx.close()
