"""Component selection in one block against NumPy on both sides of its size limit, exactly."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 31, 1023, 1024, 1025, 8193, 32767, 32768, 32769])
def test_select_components(k):
    from imageprocessor_new_b200 import _device as dev, _lib
    import torch

    rng = np.random.default_rng(k)
    stats = rng.integers(0, 40, (k + 1, 5)).astype(np.int32)
    for lo, hi in ((5, 30), (0, 100), (50, 60)):
        rows, methods = dev.empty((k, 5), torch.int32), dev.empty((k,), torch.uint8)
        kept = dev.empty((1,), torch.int32)
        ws = dev.workspace(_lib.size("spx_select_workspace_bytes", k))
        st = dev.upload(stats)
        _lib.call("spx_select_components", st.data_ptr(), k, lo, hi, _lib.REFINE_CODES["auto"], 12.0, rows.data_ptr(),
                  methods.data_ptr(), kept.data_ptr(), ws.data_ptr(), ws.numel(), dev.stream_ptr())
        keep = np.flatnonzero((stats[1:, 4] >= lo) & (stats[1:, 4] <= hi))
        n = kept.item()
        assert n == len(keep)
        want = np.column_stack((stats[1:][keep][:, :4], keep + 1))
        np.testing.assert_array_equal(rows.cpu().numpy()[:n], want)
        small = np.maximum(want[:, 2], want[:, 3]) <= 12
        np.testing.assert_array_equal(methods.cpu().numpy()[:n], np.where(small, _lib.REFINE_CODES["logquad"],
                                                                           _lib.REFINE_CODES["edge_moment"]))
