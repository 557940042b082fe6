"""Cleaned cells do not depend on how many are asked for at a time: the whole stack (a warp per cell), cells one by one and
a few of them (cut into parts), cells of fewer pixels than a warp and of no multiple of 32, bit for bit; and against the
formula in NumPy: image - background - (model - own Gaussian), each rounded once or twice at values up to 5000, and an
own Gaussian of up to 1500 whose exponent is below 20, so 1e-10 holds with an order to spare."""

import numpy as np
import pytest

from oracle import deblend as odb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(9473, 5, 6), (9472, 1, 1), (4800, 7, 9), (300, 33, 31), (7, 130, 257), (1, 200, 211)])
def test_cleaned_cells(n, h, w):
    import torch
    from imageprocessor_new_b200 import _device as dev, _lib

    rng = np.random.default_rng(n)
    cols = int(np.ceil(np.sqrt(n)))
    H, W = -(-n // cols) * h, cols * w
    img = rng.integers(0, 4000, (H, W)).astype(np.uint16)
    model = rng.uniform(0, 900, (H, W))
    i = np.arange(n)
    boxes = np.column_stack((i % cols * w, i // cols * h, np.full(n, w), np.full(n, h))).astype(np.int32)
    yy, xx = np.indices((H, W))
    vor = (yy // h * cols + xx // w).astype(np.int32)
    vor[(vor >= n) | (rng.random((H, W)) < 0.1)] = -1
    sig = max(h, w) / 4.0 + 0.5
    par = np.column_stack((rng.uniform(100, 1500, n), rng.uniform(0, w, n), rng.uniform(0, h, n),
                           -np.log(rng.uniform(0.8, 1.2, n) * sig), rng.normal(0, 0.01, n), -np.log(np.full(n, sig))))
    img_d, model_d, vor_d, boxes_d, par_d = (dev.upload(np.ascontiguousarray(a)) for a in (img, model, vor, boxes, par))
    background = _lib.BgMap(None, None, None, 0, 0, 12.5, _lib.BG_FIXED)
    cap = max(h, w, 2)

    def clean(which):
        out = torch.full((len(which), h, w), float("nan"), dtype=torch.float64, device="cuda")
        which_d = dev.upload(np.asarray(which, np.int32))
        _lib.call("spx_clean_cells", img_d.data_ptr(), dev.dtype_code(img_d), 1.0, H, W, vor_d.data_ptr(),
                  boxes_d.data_ptr(), par_d.data_ptr(), cap, background, model_d.data_ptr(), which_d.data_ptr(),
                  len(which), h, w, out.data_ptr(), dev.stream_ptr())
        return out.cpu().numpy()

    every = clean(i)
    some = sorted({0, n // 3, n - 1})
    np.testing.assert_array_equal(clean(some), every[some])
    for j in some:
        np.testing.assert_array_equal(clean([j])[0], every[j])
    for j in some:
        a, x0, y0, u1, u2, u3 = par[j]
        dy, dx = np.indices((h, w)) - np.array([y0, x0])[:, None, None]
        aa, bb = np.exp(u1) * dx + u2 * dy, np.exp(u3) * dy
        sl = np.s_[boxes[j, 1]:boxes[j, 1] + h, boxes[j, 0]:boxes[j, 0] + w]
        r = odb.render_radius(par[j:j + 1], cap)[0]
        own = np.where((abs(dx) <= r) & (abs(dy) <= r), a * np.exp(-0.5 * (aa * aa + bb * bb)), 0.0)
        want = np.where(vor[sl] == j, img[sl] - 12.5 - (model[sl] - own), 0.0)
        np.testing.assert_allclose(every[j], want, rtol=0, atol=1e-10)
