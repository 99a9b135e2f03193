"""The tables that a job exchanges with the device.  Page-locking and unlocking can
stall every stream of a device, so a context locks memory for them at most four
times, with the second job that wants so much room, never as they grow; a job with
more chunks than they have room for, and a first job, run on plain memory."""
import os
import re

import numpy as np
import pytest

from gzippy_b200 import workloads as W

ENGINE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gzippy_b200", "csrc",
                      "engine.cu")


def test_page_locks_are_few():
    """The staging ring's and the arena's, which takes four blocks at most."""
    with open(ENGINE) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    locks = [m.start() for m in re.finditer(r"cudaMallocHost\(|cudaHostAlloc\(|cudaHostRegister\(", src)]
    assert len(locks) == 2 and src.index("struct HostPinned") < locks[0] < src.index("struct TableArena") < locks[1]
    assert "blocks[4]" in src and "kRooms[4]" in src
    assert src.count("arena.add(") == 1 and src.count(" reserve_tables(total_in / ") == 1


@pytest.mark.gpu
@pytest.mark.parametrize("fine_split", [0, 1])
def test_more_chunks_than_the_tables_hold(fine_split):
    import gzippy_b200 as G
    parts = [W.content(k % 4, 60 + k, 3 << 20) for k in range(24)]
    plain = np.concatenate(parts)
    comp = W.gzip_member(plain, 6)
    small_plain = W.content(W.MARKOV, 90, 300000)
    small = W.gzip_member(small_plain, 6)
    cx = G.Context(chunk_bytes=1024, fine_split=fine_split)
    try:
        for _ in range(3):
            assert cx.decompress(small) == small_plain.tobytes()
            assert cx.decompress(comp) == plain.tobytes()
            assert cx.stats().n_chunks > 32768
    finally:
        cx.close()
