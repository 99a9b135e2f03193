"""gzgpu_decompress_device comes after the work that the caller has put on the
default stream: the input may still be on its way when the call is made."""
import numpy as np
import pytest

from gzippy_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [4096, 3 << 20])
def test_input_still_on_its_way(size):
    import torch

    import gzippy_b200 as G
    plain = W.content(W.MARKOV, 17, size)
    comp = torch.from_numpy(W.gzip_member(plain, 6).copy()).pin_memory()
    cx = G.Context()
    try:
        for _ in range(3):
            d_in = torch.zeros(comp.numel() + 1024, dtype=torch.uint8, device="cuda")
            d_out = torch.zeros(size + 64, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            torch.cuda._sleep(50_000_000)  # about 25 ms of the default stream
            d_in[: comp.numel()].copy_(comp, non_blocking=True)
            assert cx.decompress_device(d_in.data_ptr(), comp.numel(), d_out.data_ptr(), d_out.numel()) == size
            assert np.array_equal(d_out[:size].cpu().numpy(), plain)
    finally:
        cx.close()
