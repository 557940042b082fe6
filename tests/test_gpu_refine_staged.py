"""The refiners on integer images (ROIs up to 32 x 32 px staged in shared memory) against the same
refiners on the same image as float64, which takes the general path: blob sizes on either side of 16 and
32 px ROIs, one-pixel and two-pixel-thick blobs, ROIs clipped by the image, masks that are not their box.

Weighted centroids, mask means and edges are sums of exact terms or per-pixel arithmetic: the same bits.
The log-quadratic normal equations are sums in another order: 1e-9 px, the refiners' own tolerance."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 8, 10, 11, 12, 25, 26, 27, 40)


def _scene(dtype, seed):
    rng = np.random.default_rng(seed)
    top = 250 if dtype == "uint8" else 4000
    boxes, y = [], 0
    for k, h in enumerate(SIZES):
        x = 0 if k % 3 == 0 else 5
        for w in SIZES:
            boxes.append((x, y, w, h))
            x += w + 9
        y += h + 9
    hgt, wid = y - 9 + (1 if seed else 0), max(x + w for x, _, w, _ in boxes)
    img = rng.normal(0.2 * top, 0.01 * top, (hgt, wid))
    labels = np.zeros((hgt, wid), np.int32)
    rows = []
    for k, (x, y, w, h) in enumerate(boxes):
        yy, xx = np.mgrid[:h, :w]
        cy, cx = (h - 1) / 2 + rng.uniform(-0.3, 0.3), (w - 1) / 2 + rng.uniform(-0.3, 0.3)
        r2 = ((yy - cy) / max(0.5 * h, 0.7)) ** 2 + ((xx - cx) / max(0.5 * w, 0.7)) ** 2
        m = r2 <= 1.3
        m[int(round(cy)), int(round(cx))] = True
        img[y:y + h, x:x + w] += 0.7 * top * np.exp(-0.5 * r2)
        labels[y:y + h, x:x + w][m] = k + 1
        rows.append((x, y, w, h, k + 1))
    return np.clip(np.rint(img), 0, top * 1.02).astype(dtype), labels, np.array(rows, np.int32)


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("refine", ["none", "weighted", "logquad", "edge_gradmoment"])
@pytest.mark.parametrize("pad", [0, 3])
def test_staged_rois_match_the_general_path(dtype, refine, pad):
    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    for seed in (0, 1):
        img, labels, rows = _scene(dtype, seed)
        n, code = len(rows), _lib.REFINE_CODES[refine]
        lab_d, rows_d = dev.upload(labels), dev.upload(rows)
        meth_d = dev.upload(np.full(n, code, np.uint8))
        got = []
        for image in (img, img.astype(np.float64)):
            img_d, out = dev.upload(image), dev.upload(np.zeros((n, 2)))
            _lib.call("spx_refine_selected", img_d.data_ptr(), dev.dtype_code(img_d), *labels.shape, lab_d.data_ptr(),
                      rows_d.data_ptr(), meth_d.data_ptr(), n, None, pad, code, out.data_ptr(), dev.stream_ptr())
            both = dev.upload(np.zeros((n, 2)))
            _lib.call("spx_refine_centers", img_d.data_ptr(), dev.dtype_code(img_d), *labels.shape, lab_d.data_ptr(),
                      rows_d.data_ptr(), meth_d.data_ptr(), n, pad, both.data_ptr(), dev.stream_ptr())
            got.append(out.cpu().numpy())
            np.testing.assert_array_equal(both.cpu().numpy(), got[-1])
        assert np.isfinite(got[0]).all(axis=1).mean() > 0.3
        if refine == "logquad":
            np.testing.assert_allclose(got[0], got[1], rtol=0, atol=1e-9)
        else:
            np.testing.assert_array_equal(got[0], got[1])


def test_rows_past_a_device_count_are_nan():
    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    img, labels, rows = _scene("uint16", 0)
    n = len(rows)
    img_d, lab_d, rows_d = dev.upload(img), dev.upload(labels), dev.upload(rows)
    live = dev.upload(np.array([n // 2], np.int32))
    for refine in ("weighted", "logquad", "auto", "none"):
        code = _lib.REFINE_CODES[refine]
        meth = np.where(np.arange(n) % 2, 2, 3) if refine == "auto" else np.full(n, code)
        meth_d, out = dev.upload(meth.astype(np.uint8)), dev.upload(np.full((n, 2), -7.0))  # -7: not written
        _lib.call("spx_refine_selected", img_d.data_ptr(), dev.dtype_code(img_d), *labels.shape, lab_d.data_ptr(),
                  rows_d.data_ptr(), meth_d.data_ptr(), n, live.data_ptr(), 3, code, out.data_ptr(), dev.stream_ptr())
        c = out.cpu().numpy()
        assert np.isnan(c[n // 2:]).all()
        assert np.isfinite(c[: n // 2]).any() and not (c == -7.0).any()


@pytest.mark.parametrize("w,h", [(33, 1), (7, 41), (31, 33), (64, 64), (65, 63), (190, 77)])
@pytest.mark.parametrize("refine", ["none", "weighted", "logquad", "edge_gradmoment"])
def test_large_rois_take_the_same_pixels_in_the_same_order(refine, w, h):
    """ROIs that are not staged, of integer images against the same image as float64 (the same bits) and, for the mean of
    the mask, against NumPy's exact one: pixel counts on either side of a round of 32 lanes with several labels in
    flight, masks with holes, ROIs clipped by the image."""
    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    rng = np.random.default_rng(w * h)
    H, W = h + 4, w + 5
    yy, xx = np.mgrid[:H, :W]
    r2 = ((yy - 0.48 * H) / (0.45 * H)) ** 2 + ((xx - 0.53 * W) / (0.45 * W)) ** 2
    m = (r2 <= 1.2) & (rng.random((H, W)) < 0.9)
    m[:2], m[-2:], m[:, :2], m[:, -3:] = False, False, False, False
    m[2, 2] = m[h + 1, w + 1] = True
    img = np.clip(np.rint(100 + 120 * np.exp(-r2) + rng.normal(0, 2, (H, W))), 0, 255)
    lab_d, rows_d = dev.upload(np.where(m, 7, 3).astype(np.int32)), dev.upload(np.array([[2, 2, w, h, 7]], np.int32))
    code = _lib.REFINE_CODES[refine]
    meth_d = dev.upload(np.full(1, code, np.uint8))
    for pad in (0, 9):
        got = []
        for dtype in ("uint8", "uint16", "float32", "float64"):
            img_d, out = dev.upload(img.astype(dtype)), dev.upload(np.zeros((1, 2)))
            _lib.call("spx_refine_selected", img_d.data_ptr(), dev.dtype_code(img_d), H, W, lab_d.data_ptr(),
                      rows_d.data_ptr(), meth_d.data_ptr(), 1, None, pad, code, out.data_ptr(), dev.stream_ptr())
            got.append(out.cpu().numpy())
        for g in got[:-1]:
            np.testing.assert_array_equal(g, got[-1])
        if refine == "none":
            y0, x0 = max(0, 2 - pad), max(0, 2 - pad)
            ys, xs = np.nonzero(m[y0:, x0:])
            np.testing.assert_array_equal(got[-1], [[x0 + xs.sum() / len(xs), y0 + ys.sum() / len(ys)]])


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("pad", [0, 9])
def test_logquad_does_not_depend_on_the_number_of_rows(dtype, pad):
    """The same blobs as few rows, as many, and as tables with a device count on either side of 16,384 rows: the forms with
    four and with six blocks per SM, staged regions and larger ones, bit for bit."""
    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib

    img, labels, rows = _scene(dtype, 1)
    k, code = len(rows), _lib.REFINE_CODES["logquad"]
    img_d, lab_d = dev.upload(img), dev.upload(labels)
    got = []
    for times, counted in ((1, False), (30, False), (100, True), (140, True)):
        n = k * times
        rows_d, meth_d = dev.upload(np.tile(rows, (times, 1))), dev.upload(np.full(n, code, np.uint8))
        out, live = dev.upload(np.full((n, 2), -7.0)), dev.upload(np.array([n], np.int32))
        _lib.call("spx_refine_selected", img_d.data_ptr(), dev.dtype_code(img_d), *labels.shape, lab_d.data_ptr(),
                  rows_d.data_ptr(), meth_d.data_ptr(), n, live.data_ptr() if counted else None, pad, code, out.data_ptr(),
                  dev.stream_ptr())
        got.append(out.cpu().numpy())
        np.testing.assert_array_equal(got[-1], np.tile(got[0], (times, 1)))
    assert np.isfinite(got[0]).all(axis=1).mean() > 0.3
