"""The area kernels with the cubic-spline enlargement built in (spx_half_area_spline_cd,
spx_tail_area_spline_cd) against the general kernels (spx_half_area_cd, spx_tail_area_cd) given the
same enlargement as dense operators (scipy's zoom of the unit profiles), over the forms they take:
cells and windows narrower and wider than a word of sub-pixels and than a CTA's columns, single rows
and columns, ragged and empty masks, each level, peak and threshold rule, lists that overflow.

Tolerance: the two enlargements differ by a few ulps of the cell's largest value (both are FP64 sums
of at most a few hundred terms: under 1e-13 of it), so the regions, decisions against a threshold,
are the same and metrics agree to 1e-10 relative.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ANGLES = 48


def _operator(size):
    from scipy.ndimage import zoom

    cols = []
    for i in range(size):
        e = np.zeros(size + 64)
        e[32 + i] = 1.0
        cols.append(zoom(e, 4, order=3, mode="grid-constant", grid_mode=True)[128:128 + 4 * size])
    return np.ascontiguousarray(np.stack(cols, axis=1))


def _outputs(n, columns):
    import torch

    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    b = {"centers": dev.empty((n, 2), torch.float64), "contours": dev.empty((n, ANGLES + 1, 2), torch.float64),
         "status": dev.empty((n,), torch.uint8), "metrics": dev.empty((columns, n), torch.float64),
         "center_local": dev.empty((n, 2), torch.float64), "edge_px": dev.empty((n, ANGLES), torch.float64)}
    struct = _lib.MethodOut(b["centers"].data_ptr(), b["contours"].data_ptr(), b["status"].data_ptr(),
                            b["metrics"].data_ptr(), b["center_local"].data_ptr(), b["edge_px"].data_ptr(), None, None,
                            columns, n)
    return b, struct


def _same(a, b):
    np.testing.assert_array_equal(a["status"].cpu().numpy(), b["status"].cpu().numpy())
    for key in ("metrics", "centers", "center_local", "contours", "edge_px"):
        np.testing.assert_allclose(a[key].cpu().numpy(), b[key].cpu().numpy(), rtol=1e-10, atol=1e-10, err_msg=key)


def _cells(n, hm, wm, rng):
    """Noisy blobs, the last ones flat, dark, saturated and without a mask; ragged masks."""
    y, x = np.mgrid[:hm, :wm]
    cells = np.empty((n, hm, wm))
    masks = np.empty((n, hm, wm), bool)
    for i in range(n):
        cy, cx = (hm - 1) / 2 + rng.uniform(-1, 1), (wm - 1) / 2 + rng.uniform(-1, 1)
        r = np.hypot((y - cy) / max(1.0, hm / 4), (x - cx) / max(1.0, wm / 4))
        cells[i] = 3000.0 / (1 + np.exp(6 * (r - 1))) + rng.normal(0, 60, (hm, wm))
        masks[i] = (np.abs(y - cy) <= 0.47 * hm) & (rng.random((hm, wm)) < (1.0 if i % 2 else 0.97))
    cells[n - 4] = 500.0
    cells[n - 3] = -cells[n - 3]
    cells[n - 2] = np.minimum(cells[n - 2], 1500.0)
    masks[n - 1] = False
    return cells, masks


@pytest.mark.parametrize("hm, wm", [(1, 1), (3, 5), (8, 8), (9, 33), (18, 18), (24, 24), (31, 32), (33, 30), (36, 36), (2, 60)])
@pytest.mark.parametrize("median, n_top, outlines", [(1, 64, 1), (0, 7, 0), (0, 1 << 20, 1)])
def test_half_area_spline_matches_the_dense_operators(hm, wm, median, n_top, outlines):
    import torch

    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    rng = np.random.default_rng(100 * hm + wm)
    n = 9
    cells, masks = _cells(n, hm, wm, rng)
    vor = np.where(masks, np.arange(n)[:, None, None], -1).astype(np.int32).reshape(n * hm, wm)
    boxes = np.column_stack((np.zeros(n), np.arange(n) * hm, np.full(n, wm), np.full(n, hm))).astype(np.int32)
    roi = dev.upload(np.where(masks, cells, 0.0))
    vor_d, boxes_d = dev.upload(vor), dev.upload(boxes)
    zy, zx = dev.upload(_operator(hm)), dev.upload(_operator(wm))
    n_top = min(n_top, hm * wm * 16)
    got, want = [], []
    for dense in (False, True):
        (s, ss), (m, ms) = _outputs(n, 13), _outputs(n, 13)
        (want if dense else got).extend((s, m))
        head = (roi.data_ptr(), vor_d.data_ptr(), boxes_d.data_ptr(), None, n, hm, wm, wm, ANGLES)
        if dense:
            ws = dev.workspace(_lib.size("spx_half_area_workspace_bytes", hm, wm, 4))
            _lib.call("spx_half_area_cd", *head, zy.data_ptr(), zx.data_ptr(), 4, 0.5, median, n_top, outlines, ss, ms,
                      ws.data_ptr(), ws.numel(), dev.stream_ptr())
        else:
            _lib.call("spx_half_area_spline_cd", *head, 0.5, median, n_top, outlines, ss, ms, dev.stream_ptr())
        torch.cuda.synchronize()
    for a, b in zip(got, want):
        _same(a, b)
    if hm >= 8 and wm >= 8:
        assert (got[0]["status"].cpu().numpy() != 1).sum() >= 5  # regions were found


@pytest.mark.parametrize("side", [1, 3, 8, 21, 32, 33, 59, 64])
@pytest.mark.parametrize("n_top, outlines", [(64, 1), (3000, 0)])
def test_tail_area_spline_matches_the_dense_operators(side, n_top, outlines):
    import torch

    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    rng = np.random.default_rng(side)
    n = 8
    cells, _ = _cells(n, side, side, rng)
    y, x = np.mgrid[:side, :side]
    inside = np.ones((n, side, side), np.uint8)
    inside[0, :, : side // 3] = 0  # windows past the image's left and lower edge
    inside[1, 2 * side // 3:, :] = 0
    r = np.hypot(y - (side - 1) / 2, x - (side - 1) / 2)
    level = np.broadcast_to((r > 0.42 * side).astype(np.uint8), inside.shape).copy()
    zone = np.broadcast_to((r < 0.45 * side).astype(np.uint8), inside.shape).copy()
    level[2] = 0  # no level pixels
    up = [dev.upload(np.ascontiguousarray(a)) for a in (cells.astype(np.float32), inside, level, zone)]
    org = dev.upload(rng.integers(-3, 900, (n, 2)).astype(np.int32))
    cell_org = dev.upload(rng.integers(0, 900, (n, 2)).astype(np.int32))
    cuts = dev.upload(rng.uniform(100.0, 900.0, n))
    op = _operator(side)
    zy, zx_t = dev.upload(op), dev.upload(np.ascontiguousarray(op.T))
    n_top = min(n_top, side * side * 16)
    got, want = [], []
    for dense in (False, True):
        outs = [_outputs(n, 13) for _ in range(5)]
        (want if dense else got).extend(b for b, _ in outs)
        head = [a.data_ptr() for a in up] + [org.data_ptr(), cell_org.data_ptr(), n, side, ANGLES]
        tail = [0.2, n_top, outlines, cuts.data_ptr()] + [s for _, s in outs]
        if dense:
            ws = dev.workspace(_lib.size("spx_tail_area_workspace_bytes", side, 4, ANGLES))
            _lib.call("spx_tail_area_cd", *head, zy.data_ptr(), zx_t.data_ptr(), 4, *tail, ws.data_ptr(), ws.numel(),
                      dev.stream_ptr())
        else:
            _lib.call("spx_tail_area_spline_cd", *head, *tail, dev.stream_ptr())
        torch.cuda.synchronize()
    for a, b in zip(got, want):
        _same(a, b)


@pytest.mark.parametrize("size", [11, 24, 31, 33, 36])
def test_the_first_of_equal_peaks_is_taken(size):
    """Two equal isolated pixels, mirrored in the cell: equal peaks in exact arithmetic, whatever the last bits of either
    side's sums. The region is the first one's in row-major order, in cells and in windows."""
    import torch

    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    lo, hi = 2, size - 3
    pairs = [((y, lo), (y, hi)) for y in range(2, size - 2)] + [((lo, x), (hi, x)) for x in range(2, size - 2)]
    pairs += [((lo, lo), (hi, hi)), ((lo, hi), (hi, lo))]
    n = len(pairs)
    cells = np.zeros((n, size, size))
    for i, (a, b) in enumerate(pairs):
        cells[i][a] = cells[i][b] = 37.0 + 3.3 * i
    vor = np.repeat(np.arange(n, dtype=np.int32), size)[:, None] * np.ones((1, size), np.int32)
    boxes = np.column_stack((np.zeros(n), np.arange(n) * size, np.full(n, size), np.full(n, size))).astype(np.int32)
    roi, vor_d, boxes_d = dev.upload(cells), dev.upload(np.ascontiguousarray(vor)), dev.upload(boxes)
    (single, ss), (avg, sa) = _outputs(n, 13), _outputs(n, 13)
    _lib.call("spx_half_area_spline_cd", roi.data_ptr(), vor_d.data_ptr(), boxes_d.data_ptr(), None, n, size, size, size,
              ANGLES, 0.5, 0, 16, 1, ss, sa, dev.stream_ptr())
    win = dev.upload(cells.astype(np.float32))
    ones = dev.upload(np.ones((n, size, size), np.uint8))
    org = dev.upload(np.zeros((n, 2), np.int32))
    norm, sn = _outputs(n, 13)
    _lib.call("spx_tail_area_spline_cd", win.data_ptr(), ones.data_ptr(), ones.data_ptr(), ones.data_ptr(),
              org.data_ptr(), org.data_ptr(), n, size, ANGLES, 0.5, 16, 1, None, None, sn, None, None, None,
              dev.stream_ptr())
    torch.cuda.synchronize()
    want = np.array([(x, y) for (y, x), _ in pairs], float)
    for out in (single, avg):
        np.testing.assert_allclose(out["center_local"].cpu().numpy(), want, atol=0.3)
    np.testing.assert_allclose(norm["centers"].cpu().numpy(), want, atol=0.3)


@pytest.mark.parametrize("side", [9, 24, 33])
def test_levels_leave_nan_pixels_out(side):
    """NaN pixels (0 / 0 shares of the light where no model reaches) among the level pixels, all of them or some: the level
    is the median of the others, NaN without any, and never another window's. Such a window has no signal. The level is
    the middle value or the mean of two, as NumPy takes it: the same bits."""
    import torch

    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    rng = np.random.default_rng(side)
    n = 592 * 2  # several windows a block, one after another
    cells = rng.uniform(100, 900, (n, side, side)).astype(np.float32)
    level = (rng.random((n, side, side)) < 0.4).astype(np.uint8)
    ring = np.ones((side, side), bool)
    ring[1:-1, 1:-1] = False
    for i in range(n):
        if i % 4 == 1:
            cells[i][level[i] > 0] = np.nan
            cells[i][ring] = np.nan
        elif i % 4 == 3:
            cells[i][rng.random((side, side)) < 0.5] = np.nan
    ones = dev.upload(np.ones((n, side, side), np.uint8))
    org = dev.upload(np.zeros((n, 2), np.int32))
    win, level_d = dev.upload(cells), dev.upload(level)
    vor = dev.upload(np.ascontiguousarray(np.repeat(np.arange(n, dtype=np.int32), side)[:, None] * np.ones((1, side), np.int32)))
    boxes = dev.upload(np.column_stack((np.zeros(n), np.arange(n) * side, np.full(n, side), np.full(n, side))).astype(np.int32))
    roi = dev.upload(cells.astype(np.float64))
    op = _operator(side)
    zy, zx_t = dev.upload(op), dev.upload(np.ascontiguousarray(op.T))
    outs = [_outputs(n, 13) for _ in range(4)]
    head = (win.data_ptr(), ones.data_ptr(), level_d.data_ptr(), ones.data_ptr(), org.data_ptr(), org.data_ptr(), n, side,
            ANGLES)
    none = (None,) * 4
    ws = dev.workspace(max(_lib.size("spx_tail_area_workspace_bytes", side, 4, ANGLES),
                           _lib.size("spx_half_area_workspace_bytes", side, side, 4)))
    _lib.call("spx_tail_area_spline_cd", *head, 0.2, 16, 0, None, outs[0][1], *none, dev.stream_ptr())
    _lib.call("spx_tail_area_cd", *head, zy.data_ptr(), zx_t.data_ptr(), 4, 0.2, 16, 0, None, outs[1][1], *none, ws.data_ptr(),
              ws.numel(), dev.stream_ptr())
    cell = (roi.data_ptr(), vor.data_ptr(), boxes.data_ptr(), None, n, side, side, side, ANGLES)
    _lib.call("spx_half_area_spline_cd", *cell, 0.5, 1, 16, 0, outs[2][1], None, dev.stream_ptr())
    _lib.call("spx_half_area_cd", *cell, zy.data_ptr(), zy.data_ptr(), 4, 0.5, 1, 16, 0, outs[3][1], None, ws.data_ptr(),
              ws.numel(), dev.stream_ptr())
    torch.cuda.synchronize()
    import warnings

    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        values = cells.astype(np.float64).reshape(n, -1)
        tail = np.nanmedian(np.where(level.reshape(n, -1) > 0, values, np.nan), axis=1)
        half = np.nanmedian(np.where(ring.ravel()[None], values, np.nan), axis=1)
    for (b, _), want in zip(outs, (tail, tail, half, half)):
        np.testing.assert_array_equal(b["metrics"].cpu().numpy()[7], want)
        assert (b["status"].cpu().numpy()[1::2] == b["status"].cpu().numpy()[1]).all()
