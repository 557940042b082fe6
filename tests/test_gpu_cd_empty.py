"""measure_cds on pages without a cell to report (none found, or all at the border): every array of the full result has
the shape and type it has with cells, and no label is assigned."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metrics_only", [False, True])
@pytest.mark.parametrize("scene", ["flat", "border"])
def test_no_cells(scene, metrics_only):
    from imageprocessor_new_b200 import measure_cds

    img = np.full((70, 90), 100, np.uint16)
    if scene == "border":
        yy, xx = np.mgrid[:70, :90]
        img += (3000 * np.exp(-((yy - 1) ** 2 + (xx - 40) ** 2) / 18.0)).astype(np.uint16)
    res = measure_cds(img, methods=("gaussian", "halfmax", "half_area"), background_level=100.0, area_max=400,
                      metrics_only=metrics_only)
    assert res.seeds_xy.shape == (0, 2) and res.boxes_xywh.shape == (0, 4) and res.component_ids.shape == (0,)
    assert res.cell_labels.shape == img.shape and res.cell_labels.dtype == np.int32 and (res.cell_labels == -1).all()
    assert res.cell_areas_px2.shape == (0,) and res.cell_areas_px2.dtype == np.int64
    assert res.mean_intensity.shape == (0,) and res.mean_intensity.dtype == np.float64
    assert res.masks.dtype == bool and res.masks.ndim == 3 and res.masks.shape == res.rois.shape and len(res.rois) == 0
    assert (res.deblend_model["params"].shape[0] > 0) == (scene == "border")
    for m in res.measurements.values():
        assert m.centers_xy.shape == (0, 2) and m.status.shape == (0,)
