"""Members of awkward sizes back to back: the CRC pass cuts each member into
64 KiB blocks that end on 16-byte boundaries of the output, slices of 128 bytes
per thread; the marker pass looks sources up across chunks of any length.
Byte-exact, and every member's CRC and ISIZE is really checked."""
import struct
import zlib

import numpy as np
import pytest

from gzippy_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [1, 15, 16, 17, 127, 128, 129, 2047, 2049, 65519, 65520, 65535, 65536, 65537, 65552, 131072,
         131073, 200001]


@pytest.fixture(scope="module")
def ctx():
    import gzippy_b200 as G
    c = G.Context()
    yield c
    c.close()


def _members(sizes, level=6):
    plains = [W.content(i % 4, 900 + i, n) for i, n in enumerate(sizes)]
    return plains, [W.gzip_member(p, level).tobytes() for p in plains]


@pytest.mark.parametrize("rot", range(0, len(SIZES), 3))
def test_members_back_to_back(ctx, rot):
    """Each size starts at another output alignment in each rotation."""
    plains, comps = _members(SIZES[rot:] + SIZES[:rot])
    assert ctx.decompress(b"".join(comps)) == b"".join(p.tobytes() for p in plains)


@pytest.mark.parametrize("size", SIZES)
def test_single_member(ctx, size):
    (p,), (c,) = _members([size])
    assert ctx.decompress(c) == p.tobytes()


@pytest.mark.parametrize("size", SIZES[::2])
def test_wrong_trailer_is_found(ctx, size):
    import gzippy_b200 as G
    plains, comps = _members([33, size, 70])
    crc = zlib.crc32(plains[1].tobytes()) ^ 1 << (size % 32)
    bad = comps[1][:-8] + struct.pack("<II", crc, size)
    with pytest.raises(G.GzippyError) as e:
        ctx.decompress(comps[0] + bad + comps[2])
    assert e.value.code == G.CRC_MISMATCH
    short = comps[1][:-4] + struct.pack("<I", size + 1)
    with pytest.raises(G.GzippyError) as e:
        ctx.decompress(comps[0] + short + comps[2])
    assert e.value.code == G.SIZE_MISMATCH


def test_short_chunks_hold_far_sources(ctx):
    """Chunks shorter than the window: markers follow their references through
    several chunks (text whose copies reach up to 32 KiB back)."""
    import gzippy_b200 as G
    p = W.content(W.MARKOV, 77, 3 << 20)
    c = W.encode_member(p, 6, "pigz", threads=2)   # an empty stored block every MiB
    z = zlib.compressobj(6, zlib.DEFLATED, 31)
    many = b"".join(z.compress(p[i:i + 5000].tobytes()) + z.flush(zlib.Z_SYNC_FLUSH)
                    for i in range(0, p.size, 5000)) + z.flush()
    cx = G.Context(chunk_bytes=8 << 10)
    assert cx.decompress(c) == p.tobytes()
    assert cx.decompress(np.frombuffer(many, np.uint8)) == p.tobytes()
    cx.close()
