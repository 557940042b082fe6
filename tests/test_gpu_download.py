"""Chunked downloads equal the tensors they came from (sizes around the chunk and the ring of pinned
blocks, every dtype a result has, non-contiguous and empty tensors), are ordinary writable memory, and
several threads may download at once."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["uint8", "bool", "uint16", "int32", "int64", "float32", "float64"])
def test_download_equals_the_tensor(dtype):
    import torch

    from imageprocessor_new_b200 import _device as dev

    chunk, large = (b // np.dtype(dtype).itemsize for b in (dev._DOWNLOAD_CHUNK, dev._DOWNLOAD_LARGE))
    for n in (0, 1, large - 1, large, large + 1, 9 * chunk + 17, 16 * chunk + 1, 35 * chunk - 3):
        want = (np.arange(n) % 251).astype(dtype)
        got = dev.download(torch.from_numpy(want).cuda())
        assert got.dtype == want.dtype
        np.testing.assert_array_equal(got, want)
        assert got.flags.writeable
    a = torch.arange(3000 * 2000, device="cuda").view(3000, 2000).to(getattr(torch, dtype))
    np.testing.assert_array_equal(dev.download(a.t()), a.cpu().numpy().T)


def test_downloads_from_several_threads():
    from concurrent.futures import ThreadPoolExecutor

    import torch

    from imageprocessor_new_b200 import _device as dev

    def one(seed):
        with torch.cuda.stream(torch.cuda.Stream()):
            t = torch.full((5_000_003,), seed, dtype=torch.int32, device="cuda")
            return bool((dev.download(t) == seed).all())

    with ThreadPoolExecutor(6) as pool:
        assert all(pool.map(one, range(24)))
