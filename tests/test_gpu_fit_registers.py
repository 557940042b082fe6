"""Deblending iterations with either register count: 2,550 cells take one round of all warps at 96 registers and two at 128
(four warps a block); blocks of eight warps hold as many either way and run at 128. The same bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float64"])
def test_iterations_do_not_depend_on_the_registers(dtype):
    from imageprocessor_new_b200 import _device as dev, autotune
    from imageprocessor_new_b200.deblend import Deblender, build_cells

    rng = np.random.default_rng(5)
    yy, xx = np.mgrid[7:700:14, 7:714:14]
    seeds = np.column_stack((xx.ravel(), yy.ravel())) + rng.uniform(-1, 1, (yy.size, 2))
    assert 16 * 148 < len(seeds) <= 20 * 148
    y, x = np.mgrid[:700, :714]
    img = 20.0 + rng.normal(0, 1.0, x.shape)
    for sx, sy in seeds:
        sl = np.s_[max(0, int(sy) - 9):int(sy) + 10, max(0, int(sx) - 9):int(sx) + 10]
        img[sl] += 180 * np.exp(-0.5 * ((x[sl] - sx) ** 2 + (y[sl] - sy) ** 2) / 2.2 ** 2)
    page = dev.upload(np.clip(np.rint(img), 0, 255).astype(dtype))
    rows = np.column_stack((np.rint(seeds) - 6, np.full((len(seeds), 2), 13.0), seeds))
    cells = build_cells(rows, (700, 714), 3)
    before, got = autotune.current(), []
    try:
        for warps in (4, 8, 2):
            autotune.set("fit_warps", warps)
            dbl = Deblender(page, 1.0, cells)
            params, status, _ = dbl.initial(dbl.max_iter)
            model = dbl.render(params)
            bg, _ = dbl.background_of(model, dbl.stats(params, status))
            got.append([t.cpu().numpy() for t in dbl.iteration(params, model, bg)])
    finally:
        autotune.apply(before)
    assert (got[0][1] == 0).mean() > 0.9  # fits went well
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
