"""The walk from a window marker to its byte (gzippy_b200/csrc/markers.cuh),
checked on the CPU: the header is plain C++, and tests/markers_check.cpp runs it
over members of more than 4 GiB against a 64-bit model."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_marker_walk_over_4gib():
    out = os.path.join(HERE, "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "markers_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-o", exe, "-x", "c++",
                    os.path.join(HERE, "markers_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " 0 failures" in r.stdout


@pytest.mark.gpu
def test_device_over_4gib_of_one_repetition():
    """5 GiB of a 777-byte record: every chunk but the first is all markers, and
    the last ones begin more than 4 GiB into the member.  As gzip on the device and
    as raw DEFLATE, which has no checksum, through host memory."""
    import ctypes
    import struct
    import zlib

    import numpy as np
    import torch

    import gzippy_b200 as G
    rec = np.random.default_rng(9).integers(0, 256, 777, dtype=np.uint8)
    piece = np.tile(rec, 65536).tobytes()
    first = zlib.compressobj(6, zlib.DEFLATED, -15)
    raw = [first.compress(piece) + first.flush(zlib.Z_SYNC_FLUSH)]
    again = zlib.compressobj(6, zlib.DEFLATED, -15, 8, zlib.Z_DEFAULT_STRATEGY, piece[-32768:])
    raw += [again.compress(piece) + again.flush(zlib.Z_SYNC_FLUSH)] * ((5 << 30) // len(piece))
    raw = b"".join(raw) + b"\x03\x00"
    n = ((5 << 30) // len(piece) + 1) * len(piece)
    crc = 0
    for _ in range(n // len(piece)):
        crc = zlib.crc32(piece, crc)
    head = b"\x1f\x8b\x08\x00\x00\x00\x00\x00\x00\xff"
    comp = np.frombuffer(head + raw + struct.pack("<II", crc, n & 0xFFFFFFFF), np.uint8)
    cx = G.Context()
    try:
        d_in = torch.zeros(comp.size + 1024, dtype=torch.uint8, device="cuda")
        d_in[: comp.size] = torch.from_numpy(comp.copy()).cuda()
        d_out = torch.empty(n + 64, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert cx.decompress_device(d_in.data_ptr(), comp.size, d_out.data_ptr(), d_out.numel()) == n
        d, r = cx.last_chunks()
        assert (r["out_len"][d["flags"] & 2 != 0].astype(np.uint64).cumsum() > 1 << 32).sum() > 4
        assert np.array_equal(d_out[:777].cpu().numpy(), rec)
        assert torch.equal(d_out[777:n], d_out[: n - 777])
        del d_in, d_out
        torch.cuda.empty_cache()
        src = np.frombuffer(raw, np.uint8)
        out = np.empty(n, np.uint8)
        got = ctypes.c_size_t(0)
        rc = cx._lib.gzgpu_inflate_raw(cx._h, src.ctypes.data, src.size, out.ctypes.data, n, ctypes.byref(got))
        assert rc == G.OK and got.value == n
        assert np.array_equal(out.reshape(-1, 777)[::997], np.broadcast_to(rec, (n // 777, 777))[::997])
        assert all(np.array_equal(out[a:a + (64 << 20)][777:], out[a:a + (64 << 20)][:-777])
                   for a in range(0, n, (64 << 20) - 777 * 2))
    finally:
        cx.close()
