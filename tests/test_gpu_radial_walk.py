"""Half-height and gradient edges of single cells against the oracle, over step lengths, box shapes and masks: rays
along pixel lines (symmetric discs centred on a pixel), ragged masks with corners that cut rays short, one-pixel
arms, boxes up to the longest radii of the range, both forms of the ray walk.

The edges are FP64 samples with the reference's arithmetic; the two sides differ by the order of a few FP64
additions (1e-15 of the signal), which the edge formulas amplify by at most the signal over the smallest accepted
difference of two samples (1e-6 of it here), so 1e-7 px holds with two orders to spare."""

import numpy as np
import pytest

from oracle import cd as ocd

pytestmark = pytest.mark.gpu


def _cells(rng, h, w):
    yy, xx = np.indices((h, w)).astype(float)
    out = []
    for cy, cx in (((h - 1) // 2, (w - 1) // 2), ((h - 1) / 2 + 0.31, (w - 1) / 2 - 0.27)):
        r = np.hypot(yy - cy, xx - cx)
        scale = min(h, w)
        blob = 1000.0 / (1.0 + np.exp((r - 0.25 * scale) / (0.05 * scale + 0.2)))
        masks = [np.ones((h, w), bool), r <= 0.46 * scale, (r <= 0.48 * scale) & (rng.random((h, w)) < 0.93),
                 (np.abs(yy - cy) <= 1.0) | (np.abs(xx - cx) <= 2.0)]
        for m in masks:
            for noise in (0.0, 12.0):
                out.append((blob + noise * rng.normal(size=(h, w)), m))
    flat = np.full((h, w), 50.0)
    out.append((flat, np.ones((h, w), bool)))  # no crossing, no decrease
    return out


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("h,w,step", [(7, 7, 0.1), (9, 31, 0.05), (24, 25, 0.1), (25, 24, 0.37), (33, 32, 1.0),
                                      (61, 90, 0.21)])
def test_edges_match_oracle(h, w, step, form):
    import ctypes
    from imageprocessor_new_b200 import _device as dev, _lib, cd

    rng = np.random.default_rng(h * 100 + w)
    cells = _cells(rng, h, w)
    n, n_angles = len(cells), 60
    vor = np.full((n * h, w), -1, np.int32)
    boxes = np.array([[0, i * h, w, h] for i in range(n)], np.int32)
    rois = np.zeros((n, h, w))
    for i, (roi, m) in enumerate(cells):
        vor[i * h:(i + 1) * h][m] = i
        rois[i] = np.where(m, roi, 0.0)
    rois_d, vor_d, boxes_d = dev.upload(rois), dev.upload(vor), dev.upload(boxes)
    which = dev.upload(np.arange(n, dtype=np.int32))
    hb, gb = (cd._method_buffers(n, n_angles, m, True) for m in ("halfmax", "gradient"))
    before = ctypes.c_int(0)
    _lib.call("spx_tune_get", b"radial_rays", ctypes.byref(before))
    try:
        _lib.call("spx_tune_set", b"radial_rays", form)
        ws = dev.workspace(_lib.size("spx_radial_workspace_bytes", h, w, 0))
        _lib.call("spx_radial_cd", rois_d.data_ptr(), vor_d.data_ptr(), boxes_d.data_ptr(), which.data_ptr(), n, h, w,
                  w, n_angles, step, None, 0, hb[1], gb[1], ws.data_ptr(), ws.numel(), dev.stream_ptr())
    finally:
        _lib.call("spx_tune_set", b"radial_rays", before.value)
    ref = ocd.measure_cells(rois, [m for _, m in cells], np.zeros((n, 2)), np.zeros((n, 2)),
                            methods=("halfmax", "gradient"), n_angles=n_angles, radial_step=step)
    for name, b in (("halfmax", hb[0]), ("gradient", gb[0])):
        got, want = b["edge_px"].cpu().numpy(), ref[name]["edge_px"]
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want), err_msg=name)
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-7, err_msg=name)


@pytest.mark.parametrize("h,w,step", [(40, 40, 0.1), (131, 140, 0.37), (200, 211, 0.1)])
def test_edges_of_large_cells_match_oracle(h, w, step):
    """Boxes in the global scratch and noise-free cells, where most gradient maxima are walked again in FP64. A 200 px cell's
    decreases differ by 1e-6 of the signal a step around their maximum, so the bound above holds here too."""
    test_edges_match_oracle(h, w, step, 2)
