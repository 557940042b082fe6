"""Cells of several pages queued together against the same pages one by one and against the rows selected on the host,
exactly: pages without components, ones filtered out entirely, rescaled types, groups of one and of all."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pages_cells(monkeypatch):
    import torch
    from imageprocessor_new_b200 import _device as dev, synthetic, warmstart as ws
    from imageprocessor_new_b200.cd import _segment

    a = synthetic.page_square(1, shape=(160, 200)).image
    pages = [a, synthetic.page_square(2, shape=(97, 131)).image, np.zeros((40, 50), np.uint16), a.astype(np.float32),
             (a >> 4).astype(np.uint8), np.where(a > 2500, 60000, 100).astype(np.uint16)[:30, :30]]
    pages_d = [dev.upload(np.ascontiguousarray(p)) for p in pages]
    alone = [ws.page_cells(p, area_min=20, area_max=300) for p in pages_d]
    together = list(ws.pages_cells(pages_d, area_min=20, area_max=300))
    monkeypatch.setattr(ws, "_TOGETHER_PIXELS", pages[0].size + pages[1].size)
    grouped = list(ws.pages_cells(pages_d, area_min=20, area_max=300))
    assert len(together) == len(grouped) == len(pages)
    for p, one, *others in zip(pages_d, alone, together, grouped):
        comp, _ = _segment(p, "otsu", False)
        stats, cents = comp.stats.cpu().numpy()[1:].astype(np.int64), comp.centroids.cpu().numpy()[1:]
        keep = (stats[:, 4] >= 20) & (stats[:, 4] <= 300)
        np.testing.assert_array_equal(one.rows, np.column_stack((stats[:, :4], cents)).astype(np.float64)[keep])
        for c in others:
            assert (c.n, c.hm, c.wm, c.max_px) == (one.n, one.hm, one.wm, one.max_px)
            np.testing.assert_array_equal(c.rows, one.rows)
            np.testing.assert_array_equal(c.origins, one.origins)
            np.testing.assert_array_equal(c.sizes, one.sizes)
            for x, y in ((c.voronoi, one.voronoi), (c.boxes, one.boxes), (c.counts, one.counts), (c.caps, one.caps),
                         (c.seeds_d, one.seeds_d)):
                assert torch.equal(x, y)
    assert alone[2].n == 0


@pytest.mark.parametrize("limits", [(20.5, 30.5), (20, float("inf")), (float("-inf"), 300), (0, 2**40), (-3, 25.0),
                                    (2**33, 2**34), (40.2, 40.8), (300, 20), (float("nan"), 300), (20, float("nan")),
                                    (np.float32(20.5), np.int64(300))])
def test_area_limits_are_compared_as_given(limits):
    from imageprocessor_new_b200 import _device as dev, synthetic, warmstart as ws
    from imageprocessor_new_b200.cd import _segment

    page = dev.upload(synthetic.page_square(1, shape=(160, 200)).image)
    comp, _ = _segment(page, "otsu", False)
    area = comp.stats.cpu().numpy()[1:, 4]
    assert len(np.unique(area)) > 3
    got = ws.page_cells(page, area_min=limits[0], area_max=limits[1])
    keep = (area >= limits[0]) & (area <= limits[1])
    np.testing.assert_array_equal(got.rows[:, 4:6], comp.centroids.cpu().numpy()[1:][keep])
