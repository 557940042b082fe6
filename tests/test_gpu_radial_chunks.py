"""The radial methods measured and downloaded in chunks of cells against one launch, exactly."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("methods", [("halfmax", "gradient"), ("gradient",), ("gaussian", "halfmax")])
@pytest.mark.parametrize("summary", [True, False])
def test_radial_chunks(methods, summary, monkeypatch):
    from imageprocessor_new_b200 import cd, measure_cds, synthetic

    img = synthetic.page_square(5, shape=(256, 320)).image
    kw = dict(methods=methods, threshold="otsu", seeds="threshold", summary_only=summary, backend="gpu", n_angles=48,
              area_max=400)
    one = measure_cds(img, **kw)
    assert len(cd._radial_chunks(len(one.seeds_xy), 8 * 48)) == 1
    monkeypatch.setattr(cd, "_RADIAL_CHUNK", 4096)
    assert len(cd._radial_chunks(len(one.seeds_xy), 8 * 48)) > 1
    many = measure_cds(img, **kw)
    for m in methods:
        a, b = one.measurements[m], many.measurements[m]
        np.testing.assert_array_equal(a.centers_xy, b.centers_xy)
        np.testing.assert_array_equal(a.contours_xy, b.contours_xy)
        np.testing.assert_array_equal(a.status, b.status)
        for key in a.metrics:
            np.testing.assert_array_equal(a.metrics[key], b.metrics[key])
        for key in (a.geometry or {}):
            np.testing.assert_array_equal(a.geometry[key], b.geometry[key])


@pytest.mark.parametrize("n,row_bytes", [(1, 8), (10, 1 << 30), (116281, 2048), (116281, 1024), (70000, 1024)])
def test_chunk_ranges_cover_every_cell(n, row_bytes):
    from imageprocessor_new_b200 import cd

    chunks = cd._radial_chunks(n, row_bytes)
    assert 1 <= len(chunks) <= 8 and chunks[0][0] == 0 and chunks[-1][1] == n
    assert all(a[1] == b[0] for a, b in zip(chunks[:-1], chunks[1:]))
