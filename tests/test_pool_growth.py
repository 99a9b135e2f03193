"""Raw DEFLATE of a high ratio outgrows the first page pool, which is sized for
four times the input.  A chunk that runs out of pages says how far it got, in output
and input, and the pool grows by that: once, or twice where the beginning misleads."""
import ctypes
import zlib

import numpy as np
import pytest

from gzippy_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,size,chunk_bytes,most", [
    ("zeros", 256 << 20, 0, 2), ("zeros", 64 << 20, 0, 2), ("zeros", 64 << 20, 1 << 20, 2), ("runs", 64 << 20, 0, 2),
    # the last, short chunks leave most of their pages empty: the first pool does
    ("runs", 64 << 20, 4096, 0),
    # chunks decoded again after a false start grow the pool once more each
    ("record", 64 << 20, 0, 6)])
def test_pool_grows_in_few_steps(name, size, chunk_bytes, most):
    import gzippy_b200 as G
    plain = {"zeros": lambda: bytes(size), "runs": lambda: W.content(W.RUNS, 5, size).tobytes(),
             "record": lambda: (np.random.default_rng(2).integers(0, 256, 100, dtype=np.uint8).tobytes()
                                * (size // 100 + 1))[:size]}[name]()
    c = zlib.compressobj(6, zlib.DEFLATED, -15)
    comp = np.frombuffer(c.compress(plain) + c.flush(), np.uint8)
    cx = G.Context(chunk_bytes=chunk_bytes)  # a fresh pool
    try:
        out = np.empty(size, np.uint8)
        got = ctypes.c_size_t(0)
        assert cx._lib.gzgpu_inflate_raw(cx._h, comp.ctypes.data, comp.size, out.ctypes.data, size,
                                         ctypes.byref(got)) == G.OK
        assert got.value == size and out.tobytes() == plain
        assert cx.stats().pool_regrows <= most
    finally:
        cx.close()
