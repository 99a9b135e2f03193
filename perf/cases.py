"""Timed cases: what users of this package have it decode.

A case names one call of the public API and the data it is given.

* ``decompress``, ``zlib``: one stream held in host memory, ``bytes`` in and
  ``bytes`` out (``Context.decompress``, ``Context.inflate_zlib``).
* ``into``: one stream from host memory into a buffer that the caller keeps
  (``Context.decompress_into``).
* ``batch``: many host streams in one call (``Context.decompress_batch``).
* ``device``: one stream that is in device memory already and is decoded
  there (``Context.decompress_device``).
* ``batch_device``: many streams in device memory, one call
  (``Context.decompress_batch_device``).

Contents and encoder come from ``gzippy_b200.workloads``: order-2 Markov text
with copies (about 2.9 bytes out per byte in), random bytes (stored blocks),
byte runs (about 14) and noisy 16-bit ramps (about 1.02); ``mixed`` cycles all
four in segments.  Levels 6 and 9 write dynamic Huffman blocks, level 1 fixed
ones.  Every member is one serial zlib stream without flush seams.

All cases share one Context, as a program's calls do.
"""
import os
import zlib
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import gzippy_b200 as G
from gzippy_b200 import workloads as W

KINDS = {"text": W.MARKOV, "random": W.RANDOM, "runs": W.RUNS, "ramps": W.RAMPS}
# compressed bytes per plain byte at level 6 (16 MiB of each; level 1 of text is 0.47)
RATIO = {"text": 0.35, "random": 1.0, "runs": 0.073, "ramps": 0.98, "mixed": 0.60}
KIB, MIB = 1 << 10, 1 << 20

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = G.Context()
    return _ctx


def listed():
    return [
        # the smallest call: a web response or a small file, all latency
        {"name": "host_text_4k", "call": "decompress", "content": "text", "bytes": 4 * KIB, "level": 6},
        # a zlib chunk as object stores and image files hold them, an odd size
        {"name": "host_zlib_text_100k", "call": "zlib", "content": "text", "bytes": 100001, "level": 6},
        # an ordinary file, every kind of block in it
        {"name": "host_mixed_3m", "call": "decompress", "content": "mixed", "bytes": 3 * MIB + 1234,
         "level": 6, "segment": 256 * KIB},
        # a large file of 24 members from host memory into the caller's buffer: copies both ways and the decode
        {"name": "host_members_48m", "call": "into", "content": "mixed", "bytes": 48 * MIB + 77, "level": 6,
         "segment": 1 * MIB, "members": 24},
        # requests of a service, 4 to 256 KiB each, merged into one call
        {"name": "host_requests_64", "call": "batch", "streams": 64, "low": 4 * KIB, "high": 256 * KIB},
        # one record shard in device memory, few blocks, an odd size
        {"name": "device_text_1m", "call": "device", "content": "text", "bytes": 1000003, "level": 6},
        # numeric samples: literal codes nearly all of one length, hardly a match
        {"name": "device_ramps_12m", "call": "device", "content": "ramps", "bytes": 12 * MIB + 5, "level": 6},
        # fixed Huffman codes (the fast level): no block headers to start at
        {"name": "device_text_l1_16m", "call": "device", "content": "text", "bytes": 16 * MIB, "level": 1},
        # highly compressible data at the best level: the output side
        {"name": "device_runs_l9_64m", "call": "device", "content": "runs", "bytes": 64 * MIB + 4097, "level": 9},
        # the text stream of the workload list
        {"name": "device_text_64m", "call": "device", "content": "text", "bytes": 64 * MIB, "level": 6},
        # the 4 MiB segments of the headline stream, as one member
        {"name": "device_mixed_128m", "call": "device", "content": "mixed", "bytes": 128 * MIB, "level": 6,
         "segment": 4 * MIB},
        # many independent streams, log-normal sizes (median 64 KiB), all kinds and levels
        {"name": "device_batch_600", "call": "batch_device", "streams": 600, "low": KIB, "high": 16 * MIB},
    ]


def _log(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    call = rng.choice(["decompress", "zlib", "into", "batch", "device", "device", "device", "batch_device"])
    if call == "batch":
        return {"call": call, "streams": _log(rng, 2, 200), "low": 4 * KIB, "high": 256 * KIB}
    if call == "batch_device":
        return {"call": call, "streams": _log(rng, 8, 600), "low": KIB, "high": _log(rng, 64 * KIB, 16 * MIB)}
    low, high = {"decompress": (KIB, 8 * MIB), "zlib": (KIB, 4 * MIB), "into": (256 * KIB, 48 * MIB),
                 "device": (16 * KIB, 64 * MIB)}[call]
    case = {"call": call, "content": rng.choice(["text", "random", "runs", "ramps", "mixed", "mixed"]),
            "bytes": _log(rng, low, high), "level": rng.choice([1, 6, 6, 9])}
    if case["content"] == "mixed":
        case["segment"] = _log(rng, 16 * KIB, 4 * MIB)
    if call in ("device", "into") and rng.random() < 0.3:  # members of one size back to back, as parallel writers leave them
        case["members"] = rng.randrange(2, 33)
    return case


def _plain(content, seed, n, segment=0):
    if content != "mixed":
        return W.content(KINDS[content], seed, n)
    out = np.empty(n, np.uint8)

    def fill(i):
        a = i * segment
        b = min(n, a + segment)
        out[a:b] = W.content(i % 4, seed * 1000003 + i, b - a)

    with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
        list(ex.map(fill, range(-(-n // segment))))
    return out


def _stream(case, seed):
    """(compressed, plain size): one gzip stream of one or several members."""
    members = case.get("members", 1)
    plain = _plain(case["content"], seed, case["bytes"], case.get("segment", 0))
    parts = np.array_split(plain, members)
    with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
        return np.concatenate(list(ex.map(lambda p: W.gzip_member(p, case["level"]), parts))), plain.size


def _specs(case):
    """(size, content, level) of every stream: the case's own, the same for every seed."""
    n = case["streams"]
    rng = np.random.default_rng(n)
    if case["call"] == "batch":  # log-uniform, the small requests of the serving workload
        sizes = np.exp(rng.uniform(np.log(case["low"]), np.log(case["high"]), n)).astype(np.int64)
    else:
        sizes = W.lognormal_sizes(rng, n, lo=case["low"], hi=case["high"])
    return sizes, rng.integers(0, 4, n), rng.choice([1, 6, 9], n)


def _streams(case, seed):
    sizes, kinds, levels = _specs(case)

    def one(i):
        return W.gzip_member(W.content(int(kinds[i]), seed * 104729 + i, int(sizes[i])), int(levels[i]))

    with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
        return list(ex.map(one, range(sizes.size))), sizes


def prepare(case, seed):
    call = case["call"]
    state = {"call": call, "ctx": _context()}
    if call in ("batch", "batch_device"):
        comps, sizes = _streams(case, seed)
        total = int(sizes.sum())
        if call == "batch":
            state["data"] = [c.tobytes() for c in comps]
            return state
        # offsets on 16-byte boundaries, readable bytes after the last stream
        lens = np.array([c.size for c in comps], np.uint64)
        offs = np.concatenate([[0], np.cumsum((lens + np.uint64(15)) & ~np.uint64(15))]).astype(np.uint64)
        packed = np.zeros(int(offs[-1]) + 1024, np.uint8)
        for o, c in zip(offs, comps):
            packed[int(o):int(o) + c.size] = c
        state.update(offs=offs[:-1], lens=lens, src=torch.from_numpy(packed).cuda(),
                     dst=torch.empty(total, dtype=torch.uint8, device="cuda"))
        return state
    if call == "zlib":
        plain = _plain(case["content"], seed, case["bytes"], case.get("segment", 0))
        state["data"] = zlib.compress(plain.tobytes(), case["level"])
        return state
    comp, n = _stream(case, seed)
    if call == "device":
        src = torch.zeros(comp.size + 1024, dtype=torch.uint8)
        src[:comp.size] = torch.from_numpy(comp)
        state.update(src=src.cuda(), size=comp.size, dst=torch.empty(n, dtype=torch.uint8, device="cuda"))
    elif call == "into":
        state.update(data=comp, dst=np.empty(n, np.uint8))
    else:
        state["data"] = comp.tobytes()
    return state


def run(state):
    ctx, call = state["ctx"], state["call"]
    if call == "decompress":
        return np.frombuffer(ctx.decompress(state["data"]), np.uint8)
    if call == "zlib":
        return np.frombuffer(ctx.inflate_zlib(state["data"]), np.uint8)
    if call == "into":
        return state["dst"][:ctx.decompress_into(state["data"], state["dst"])]
    if call == "batch":
        outs = ctx.decompress_batch(state["data"])
        return np.frombuffer(b"".join(outs), np.uint8)
    dst = state["dst"]
    if call == "device":
        n = ctx.decompress_device(state["src"].data_ptr(), state["size"], dst.data_ptr(), dst.numel())
        return dst[:n]
    offs, lens, _ = ctx.decompress_batch_device(state["src"].data_ptr(), state["offs"], state["lens"],
                                                dst.data_ptr(), dst.numel())
    return dst, offs.astype(np.int64), lens.astype(np.int64)


def work(case):
    """The compressed bytes read once and the plain bytes written once."""
    if "streams" in case:
        sizes, kinds, _ = _specs(case)
        plain = int(sizes.sum())
        ratio = sum(RATIO[k] * int(sizes[kinds == v].sum()) for k, v in KINDS.items()) / plain
    else:
        plain, ratio = case["bytes"], RATIO[case["content"]]
    return {"bytes": int(plain * (1 + ratio)), "flops": 0}
