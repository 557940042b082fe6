"""CDResult.mean_intensity: the sums over each cell's pixels, in raster order, as gathering the assigned
pixels first gives them (the same bits), for every image type and with pixels of no cell."""

import numpy as np
import pytest

from imageprocessor_new_b200.types import CDResult


@pytest.mark.parametrize("dtype", ["uint8", "uint16", "int64", "float32", "float64"])
@pytest.mark.parametrize("cells", [0, 1, 7])
def test_mean_intensity_matches_the_gathered_sums(dtype, cells):
    rng = np.random.default_rng(cells)
    image = (rng.random((37, 41)) * 200).astype(dtype)
    labels = rng.integers(-1, max(cells, 1), (37, 41)).astype(np.int32) if cells else np.full((37, 41), -1, np.int32)
    assigned = labels >= 0
    areas = np.bincount(labels[assigned], minlength=cells)
    want = np.bincount(labels[assigned], weights=image[assigned].astype(np.float64), minlength=cells)
    want = np.divide(want, areas, out=np.full(cells, np.nan), where=areas > 0)
    empty = np.zeros((cells, 0))
    res = CDResult(image=image, binary=image > 0, component_labels=labels, component_ids=np.zeros(cells, int),
                   boxes_xywh=empty, seeds_xy=np.zeros((cells, 2)), cell_labels=labels, cell_areas_px2=areas,
                   origins_xy=empty, rois=empty, masks=empty, measurements={})
    np.testing.assert_array_equal(res.mean_intensity, want)


def _result(image, labels, cells, areas):
    empty = np.zeros((cells, 0))
    return CDResult(image=image, binary=image > 0, component_labels=labels, component_ids=np.zeros(cells, int),
                    boxes_xywh=empty, seeds_xy=np.zeros((cells, 2)), cell_labels=labels, cell_areas_px2=areas,
                    origins_xy=empty, rois=empty, masks=empty, measurements={})


@pytest.mark.parametrize("dtype", ["int8", "int16", "int32", "int64", "uint8", "uint16", "uint32"])
def test_every_negative_label_is_a_pixel_of_no_cell(dtype):
    """Labels below -1 too, and labels up to the top of their type (none wraps round)."""
    rng = np.random.default_rng(0)
    info = np.iinfo(dtype)
    cells = min(int(info.max), 300) + 1
    labels = rng.integers(max(int(info.min), -200), cells, (37, 41)).astype(dtype)
    labels[0, :3] = cells - 1
    image = rng.random((37, 41))
    image[labels.astype(np.int64) < 0] = np.nan
    assigned = labels >= 0
    areas = np.bincount(labels[assigned], minlength=cells)
    want = np.bincount(labels[assigned], weights=image[assigned], minlength=cells)
    want = np.divide(want, areas, out=np.full(cells, np.nan), where=areas > 0)
    np.testing.assert_array_equal(_result(image, labels, cells, areas).mean_intensity, want)


@pytest.mark.parametrize("shape", [(41, 37), (37 * 41,), (37, 41, 1)])
def test_an_image_of_another_shape_is_refused(shape):
    with pytest.raises(IndexError):
        _result(np.ones(shape), np.zeros((37, 41), np.int32), 1, np.array([37 * 41]))
