"""The CRC pass's blocks as the host cuts them (gzippy_b200/csrc/engine.cu), on the
CPU against zlib: they end on 16-byte boundaries of the output, the last one at or
past its member's end, slices are counted back from a block's end, bytes outside the
member count as zeros, and the member's check takes the zeros after it back with
x^(8 (2^32 - 1 - pad)), since x^(2^32 - 1) = 1 mod P."""
import random
import zlib

import pytest

from test_crc_model import mulmod, raw_crc, x_pow_8n

SLICE, THREADS = 128, 512  # kCrcSlice, kCrcThreads
BLOCK = SLICE * THREADS    # kCrcBlock


def member_crc(out: bytes, moff: int, m1: int) -> int:
    end = (m1 + 15) & ~15
    blocks, e = [], end
    while e > moff:
        b = e - BLOCK if e > moff + BLOCK else moff
        if b < m1:
            blocks.append((b, min(e, m1), e, end - e))
        if b == moff:
            break
        e = b
    random.Random(m1).shuffle(blocks)
    acc = 0
    for begin, last, e, after in blocks:
        reg = 0
        for t in range(THREADS):  # slices in order: each moves what is before it on
            s0 = e - SLICE * (THREADS - t)
            if s0 + SLICE <= begin:
                continue
            data = bytes(out[a] if begin <= a < last else 0 for a in range(s0, s0 + SLICE))
            reg = mulmod(x_pow_8n(SLICE), reg) ^ raw_crc(data)
        acc ^= mulmod(x_pow_8n(after), reg)
    pad = -m1 & 15
    if pad:
        acc = mulmod(x_pow_8n(0xFFFFFFFF - pad), acc)
    return ~(mulmod(x_pow_8n(m1 - moff), 0xFFFFFFFF) ^ acc) & 0xFFFFFFFF


@pytest.mark.parametrize("moff,n", [(0, 0), (0, 1), (5, 11), (0, 16), (3, 13), (3, 14), (16, 4096), (7, 65536),
                                    (0, 65536), (0, 65537), (9, 65535), (15, 131073), (1, 70001)])
def test_member_crc_with_padded_end(moff, n):
    out = bytes(random.Random(n).getrandbits(8) for _ in range(moff + n + 40))  # other members around it
    assert member_crc(out, moff, moff + n) == zlib.crc32(out[moff:moff + n])


def test_taking_zeros_back():
    for pad in range(1, 16):
        assert mulmod(x_pow_8n(0xFFFFFFFF - pad), x_pow_8n(pad)) == 1 << 31
