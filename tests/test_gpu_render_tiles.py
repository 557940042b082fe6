"""The model render with every tile edge it can be set to, bit for bit against one another and against the oracle:
pages where each edge is kept (592 tiles of 64 px and more), with sides that are no multiples of it, and pages where
the size rule takes a smaller one. The model's buffer holds NaN before, so that a pixel nobody writes shows.

Against the oracle: a term is at most 1000 and its exponent at most some tens, so the two sides' exponent and
exponential roundings (a few 1e-16 relative each, times the exponent) stay below 2e-11 a term; at most 50 Gaussians cover
a pixel, so 1e-9 holds for their sum."""

import numpy as np
import pytest

from oracle import deblend as odb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(2047, 1601), (1600, 1600), (1281, 2049), (700, 900), (33, 65), (1, 1)])
def test_every_tile_edge_renders_the_same_model(h, w):
    import torch
    from imageprocessor_new_b200 import _device as dev, _lib, autotune

    rng = np.random.default_rng(h + w)
    n, cap = max(40, min(1200, h * w // 400)), 40
    local = np.column_stack((rng.uniform(10, 1000, n), rng.uniform(-2, 9, n), rng.uniform(-2, 9, n),
                             -np.log(rng.uniform(0.7, 9.0, n)), rng.normal(0, 0.02, n), -np.log(rng.uniform(0.7, 9.0, n))))
    boxes = np.column_stack((rng.integers(-8, w + 2, n), rng.integers(-8, h + 2, n), np.full(n, 8), np.full(n, 8)))
    params_d, boxes_d = dev.upload(local), dev.upload(boxes.astype(np.int32))
    ws = dev.workspace(_lib.size("spx_render_workspace_bytes", n, h, w))
    before = autotune.get("render_tile")
    got = {}
    try:
        for tile in autotune.KNOBS["render_tile"]:
            autotune.set("render_tile", tile)
            model = dev.empty((h, w), torch.float64).fill_(float("nan"))
            _lib.call("spx_render_model", params_d.data_ptr(), boxes_d.data_ptr(), n, h, w, cap, model.data_ptr(),
                      ws.data_ptr(), ws.numel(), dev.stream_ptr())
            got[tile] = model.cpu().numpy()
    finally:
        autotune.set("render_tile", before)
    for tile, model in got.items():
        np.testing.assert_array_equal(model, got[16], err_msg=str(tile))
    glob = local.copy()
    glob[:, 1:3] += boxes[:, :2]
    np.testing.assert_allclose(got[64], odb.render(glob, (h, w), cap), rtol=0, atol=1e-9)
