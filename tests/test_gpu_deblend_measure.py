"""The deblending loop's one read-back (spx_deblend_measure) against its separate parts: the same statistics and the
same tile medians and counts, exactly (both sides select and average the same values with the same roundings)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tile,excluded", [(np.uint16, 64, False), (np.uint8, 50, True), (np.float32, 37, True),
                                                 (np.float64, 256, False)])
def test_measure_matches_its_parts(dtype, tile, excluded):
    import torch
    from imageprocessor_new_b200 import _device as dev, _lib, synthetic
    from imageprocessor_new_b200.deblend import Deblender
    from imageprocessor_new_b200.warmstart import page_cells

    page = synthetic.page_square(3, shape=(200, 231)).image
    img = (page >> 4).astype(dtype) if np.dtype(dtype) == np.uint8 else page.astype(dtype)
    img_d = dev.upload(img)
    cells = page_cells(dev.upload(page))
    exclude = None
    if excluded:
        e = np.zeros(img.shape, np.uint8)
        e[:70, 40:160] = 1
        exclude = dev.upload(e)
    d = Deblender(img_d, 1.0, cells, exclude_d=exclude, tile=tile)
    params, status, _ = d.initial(10)
    model = d.render(params)
    rng = np.random.default_rng(0)
    steps = rng.random(cells.n)
    steps[::5] = np.nan
    none_ok = torch.full_like(status, 3)
    no_steps = dev.upload(np.full(cells.n, np.inf))
    for st, ms, usable in ((status, None, False), (status, dev.upload(steps), True), (none_ok, no_steps, True)):
        stats, (free, count, use) = d.measure(model, params, st, ms, usable)
        want = d.stats(params, st, ms)
        np.testing.assert_array_equal(stats, want)
        med, cnt = d._tile_medians(model, _lib.TILE_FREE, d.free_fraction * want[0], d.free_distance_fwhm * want[1])
        np.testing.assert_array_equal(free, med)
        np.testing.assert_array_equal(count, cnt)
        assert (use is not None) == usable
        if usable:
            np.testing.assert_array_equal(use, d._tile_medians(model, _lib.TILE_USABLE)[0])
    fixed = Deblender(img_d, 1.0, cells, tile=tile, background_level=3.0)
    stats, medians = fixed.measure(model, params, status)
    assert medians is None
    np.testing.assert_array_equal(stats, fixed.stats(params, status))
