"""Barriers of a CTA are those of gzippy_b200/csrc/barrier.cuh, which join each
warp's lanes first: lanes leave the decoder's data-dependent loops at different
times, and a warp whose lanes reach a CTA's barrier apart is undefined."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gzippy_b200", "csrc")


def test_no_bare_cta_barrier():
    bare = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        if os.path.basename(path) == "barrier.cuh":
            continue
        with open(path) as f:
            for i, line in enumerate(f, 1):
                if re.search(r"__syncthreads|bar(rier)?\.sync", line.split("//")[0]):
                    bare.append(f"{os.path.basename(path)}:{i}")
    assert not bare
