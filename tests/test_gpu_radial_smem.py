"""Radial profiles at the box sizes whose shared memory passes 48 KB only together with the kernel's static arrays: the
launch succeeds, and a constant-background disc gives the same half-height radius from every ray to a tenth of a pixel."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,smooth", [(24, 24, True), (22, 26, True), (12, 44, True), (25, 38, False), (34, 29, False),
                                         (16, 55, False)])
def test_launches(h, w, smooth):
    from imageprocessor_new_b200 import _device as dev, _lib, cd
    from imageprocessor_new_b200.peaks import gaussian_weights

    bytes_ = _lib.size("spx_radial_workspace_bytes", h, w, int(smooth))
    assert bytes_ == 256  # the cell fits shared memory
    yy, xx = np.indices((h, w)).astype(float)
    r = np.hypot(yy - (h - 1) / 2, xx - (w - 1) / 2)
    roi = 1000.0 / (1.0 + np.exp((r - 0.25 * min(h, w)) / 1.0))
    args = (dev.upload(roi), dev.upload(np.zeros((h, w), np.int32)), dev.upload(np.array([[0, 0, w, h]], np.int32)))
    hb = cd._method_buffers(1, 64, "halfmax", True)
    weights, radius = gaussian_weights(0.5)
    weights_d = dev.upload(weights) if smooth else None
    ws = dev.workspace(bytes_)
    _lib.call("spx_radial_cd", *(a.data_ptr() for a in args), None, 1, h, w, w, 64, 0.1, dev.ptr(weights_d),
              radius if smooth else 0, hb[1], None, ws.data_ptr(), ws.numel(), dev.stream_ptr())
    edge = hb[0]["edge_px"].cpu().numpy()
    assert np.isfinite(edge).all() and np.ptp(edge) < 0.1
