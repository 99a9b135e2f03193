"""The autotuner tries only what has an effect: the number of CTAs per SM has none
in jobs of up to two chunks per SM, which one CTA of 1,024 threads per SM decodes."""
import pytest

from gzippy_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,trials", [(3 << 20, 6), (96 << 20, 8)])
def test_trials(size, trials):
    """Besides the default: chunk sizes (four, of which 16 KiB is the small job's
    default), two table sizes and, in the large job, four CTAs per SM."""
    import gzippy_b200 as G
    plain = W.content(W.MARKOV, 41, size)
    comp = W.gzip_member(plain, 6)
    cx = G.Context(autotune=1)
    try:
        assert cx.decompress(comp) == plain.tobytes()
        s = cx.stats()
        if size < 8 << 20:
            assert s.tune_trials == trials and s.ctas_per_sm == 3
        else:  # (the fastest chunk size may leave two chunks per SM or fewer)
            assert s.tune_trials in (trials - 1, trials)
    finally:
        cx.close()
