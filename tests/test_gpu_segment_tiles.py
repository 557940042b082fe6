"""Labelling by one warp per 32 x 64 tile (ragged sizes, pixel types, thresholds), the Otsu scan's two routes and
the parallel triangle scan, against the oracle. Whole numbers throughout: everything is compared exactly."""

import numpy as np
import pytest

from oracle import segment as osg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32, np.float64])
@pytest.mark.parametrize("conn", [8, 4])
def test_labels_over_types_and_thresholds(dtype, conn):
    from imageprocessor_new_b200 import _device as dev, segment

    rng = np.random.default_rng(31 + conn)
    for shape in ((1, 3), (2, 66), (31, 63), (32, 64), (33, 128), (65, 194), (130, 321)):
        img = (rng.integers(0, 256, shape) if np.dtype(dtype).kind == "u" else rng.normal(100, 60, shape)).astype(dtype)
        for thr, invert in ((99.5, False), (99.0, True), (-3.0, False), (-0.5, True), (1e9, False), (1e9, True),
                            (float("nan"), False), (float("nan"), True), (float("inf"), True)):
            comp = segment.label(dev.upload(img), fixed_threshold=thr, invert=invert, connectivity=conn)
            v = img.astype(np.float64)
            num, labels, stats, cents = osg.label_components(v <= thr if invert else v > thr, conn)
            assert comp.count + 1 == num
            np.testing.assert_array_equal(comp.labels.cpu().numpy(), labels)
            keep = stats[:, 4] > 0  # an empty background has no box
            np.testing.assert_array_equal(comp.stats.cpu().numpy()[keep], stats[keep])
            np.testing.assert_array_equal(comp.centroids.cpu().numpy()[keep][1:], cents[keep][1:])


def _otsu(hist, dtype):
    import torch
    from imageprocessor_new_b200 import _device as dev, _lib

    occupied = np.nonzero(hist)[0]
    h = dev.upload(hist.astype(np.uint32).view(np.int32))
    rng = dev.upload(np.array([occupied[0], occupied[-1]], np.int32))
    out = dev.empty((1,), torch.float64)
    code = _lib.DTYPES[np.dtype(dtype)]
    ws = dev.workspace(_lib.size("spx_otsu_workspace_bytes", code))
    _lib.call("spx_otsu_from_histogram", h.data_ptr(), code, rng.data_ptr(), int(hist.sum()), out.data_ptr(),
              ws.data_ptr(), ws.numel(), dev.stream_ptr())
    return out.item()


def test_otsu_scan_both_routes():
    """Histograms the certified pick decides (a smooth valley) and those only the sequential scan does (an
    empty valley, equal variances, two or three levels, one level), over one and many chunks of 1,024 bins."""
    rng = np.random.default_rng(8)
    hists = []
    for n in (2, 3, 255, 1023, 1024, 1025, 2049, 40000, 65536):
        for lo in (0, 65536 - n):
            h = np.zeros(65536, np.int64)
            h[lo:lo + n] = rng.integers(0, 50, n)
            h[lo] = h[lo + n - 1] = 7
            hists.append(h)
            gap = h.copy()
            gap[lo + n // 3: lo + max(n - 1 - n // 3, n // 3)] = 0  # an empty run around the middle
            hists.append(gap)
            two = np.zeros(65536, np.int64)
            two[lo], two[lo + n - 1] = 1 << 31, 3  # the second class is below FLT_EPSILON
            hists.append(two)
            two = two.copy()
            two[lo + n - 1] = 123456
            hists.append(two)
    one = np.zeros(65536, np.int64)
    one[500] = 9
    hists.append(one)
    for i, h in enumerate(hists):
        assert _otsu(h, np.uint16) == osg.otsu_from_histogram(h, int(h.sum())), i
    for i in range(20):
        h = np.zeros(65536, np.int64)
        h[:256] = rng.integers(0, 1 << (1 + i), 256) * (rng.random(256) < 0.05 * (i + 1))
        h[rng.integers(0, 256)] += 5
        assert _otsu(h, np.uint8) == osg.otsu_from_histogram(h[:256], int(h.sum())), i


def test_triangle_scan_edges():
    """Peaks at both ends, plateaus, one level, few levels, both slopes."""
    from imageprocessor_new_b200 import _device as dev, segment

    rng = np.random.default_rng(4)
    images = [np.full((5, 7), v, np.uint8) for v in (0, 1, 128, 254, 255)]
    images += [np.array([[0, 255]], np.uint8), np.array([[0, 0, 255]], np.uint8), np.array([[0, 255, 255]], np.uint8)]
    images += [np.repeat(np.arange(256, dtype=np.uint8), 3)[None]]
    for mean, sd in ((20, 8), (230, 9), (128, 40), (3, 30), (252, 30)):
        images.append(np.clip(rng.normal(mean, sd, (90, 71)), 0, 255).astype(np.uint8))
    for levels in (2, 3, 9):
        images.append(rng.choice(rng.integers(0, 256, levels), (33, 40)).astype(np.uint8))
    for i, img in enumerate(images):
        assert segment.triangle(dev.upload(img)).item() == osg.triangle_threshold(img), i
