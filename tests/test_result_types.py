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
