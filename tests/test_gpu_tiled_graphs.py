"""Band graphs are reused across pages of other thresholds, grow after an overflow, and are never shared
between calls that run at the same time."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _page(seed, holes=1.0, level=1000.0):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[:700, :420]
    img = np.full((700, 420), level)
    for cy in range(12, 700, 20):
        for cx in range(12, 420, 20):
            if rng.random() < holes:
                oy, ox = rng.uniform(-1, 1, 2)
                img[cy - 9:cy + 10, cx - 9:cx + 10] += 3000 / (1 + np.exp(3 * (np.hypot(
                    y[cy - 9:cy + 10, cx - 9:cx + 10] - cy - oy, x[cy - 9:cy + 10, cx - 9:cx + 10] - cx - ox) - 4.5)))
    return np.rint(img + rng.normal(0, 15, img.shape)).astype(np.uint16)


KW = dict(threshold="otsu", refine="weighted", tile_h=256, overlap=64, threshold_mode="global", area_max=400)


def _eager(page):
    from imageprocessor_new_b200 import centers, tiled

    kw = dict(KW, invert=False, area_min=1, pad=3, connectivity=8, small_feature_max=12.0, otsu_downsample=4,
              thr_scale=0.8, dedupe_eps=1.5, device=0)
    return tiled.detect_tiled(page, use_graphs=False, **kw).centers_xy


def test_a_graph_serves_pages_of_other_thresholds(monkeypatch):
    from imageprocessor_new_b200 import detect_centers, tiled

    built = []
    init = tiled.BandGraph.__init__
    monkeypatch.setattr(tiled.BandGraph, "__init__", lambda self, *a, **k: (built.append(1), init(self, *a, **k))[1])
    tiled._GRAPHS.clear()
    for seed, level in ((0, 1000.0), (1, 1500.0), (2, 400.0)):
        page = _page(seed, level=level)
        res = detect_centers(page, backend="gpu", **KW)
        assert res.meta["band_graphs"]
        np.testing.assert_array_equal(res.centers_xy, _eager(page))
    assert len(built) == 2  # the full bands' and the last band's


def test_a_graph_grows_once_after_an_overflow(monkeypatch):
    from imageprocessor_new_b200 import detect_centers, tiled

    monkeypatch.setattr(tiled, "band_capacity", lambda h, w, c=None: 40 if c is None else 2 * int(c))
    tiled._GRAPHS.clear()
    tiled._COMPONENTS.clear()
    sparse, dense = _page(3, holes=0.1), _page(4)
    for page, graphed in ((sparse, True), (dense, False), (sparse, True), (dense, True), (sparse, True)):
        res = detect_centers(page, backend="gpu", **KW)
        assert res.meta["band_graphs"] == graphed
        np.testing.assert_array_equal(res.centers_xy, _eager(page))
    tiled._GRAPHS.clear()
    tiled._COMPONENTS.clear()


def test_calls_from_several_threads_do_not_share_a_graph():
    from concurrent.futures import ThreadPoolExecutor

    import torch

    from imageprocessor_new_b200 import detect_centers, tiled

    pages = [_page(10 + k, holes=0.5 + 0.1 * k, level=500.0 + 200 * k) for k in range(4)]
    want = [_eager(p) for p in pages]
    for p in pages:  # graphs exist before the threads start (a capture forbids other threads' allocations)
        detect_centers(p, backend="gpu", **KW)
    held = [g for idle in tiled._GRAPHS.values() for g in idle]
    assert held
    key = next(iter(tiled._GRAPHS))
    a, b = tiled._take_graph(key), tiled._take_graph(key)
    assert a is not None and b is None  # taken once only
    tiled._put_graph(key, a)

    def run(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            return detect_centers(pages[k], backend="gpu", **KW).centers_xy

    with ThreadPoolExecutor(1) as pool:  # another thread and stream than the graphs were built on
        for k, got in enumerate(pool.map(run, range(4))):
            np.testing.assert_array_equal(got, want[k])


@pytest.mark.parametrize("warm", [False, True])
def test_a_capture_leaves_overlapping_calls_alone(monkeypatch, warm):
    """While one thread captures its first graph another allocates device and pinned memory and runs whole calls, from
    an empty pool and with idle graphs of its own: both succeed with the eager path's centres."""
    import threading

    import torch

    from imageprocessor_new_b200 import detect_centers, tiled

    first, second = _page(20), _page(21, holes=0.6)[:, :380]
    want = [_eager(first), _eager(second)]
    tiled._GRAPHS.clear()
    if warm:
        detect_centers(second, backend="gpu", **KW)
    capturing, other_done, failed, got = threading.Event(), threading.Event(), [], {}
    launch = tiled.BandGraph._launch

    def slow_launch(self):
        if self.shape[1] == first.shape[1] and torch.cuda.is_current_stream_capturing() and not capturing.is_set():
            capturing.set()
            assert other_done.wait(60)
        launch(self)

    monkeypatch.setattr(tiled.BandGraph, "_launch", slow_launch)

    def capture():
        with torch.cuda.stream(torch.cuda.Stream()):
            got["first"] = detect_centers(first, backend="gpu", **KW)

    def others():
        try:
            assert capturing.wait(60)
            with torch.cuda.stream(torch.cuda.Stream()):
                held = [torch.empty(96 << 20, dtype=torch.uint8, device="cuda"),
                        torch.empty(48 << 20, dtype=torch.uint8, pin_memory=True)]
                for _ in range(3):
                    got["second"] = detect_centers(second, backend="gpu", **KW)
                del held
        finally:
            other_done.set()

    def run(fn):
        try:
            fn()
        except BaseException as e:
            failed.append(e)

    threads = [threading.Thread(target=run, args=(f,)) for f in (capture, others)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    assert capturing.is_set()
    np.testing.assert_array_equal(got["first"].centers_xy, want[0])
    np.testing.assert_array_equal(got["second"].centers_xy, want[1])
    assert got["first"].meta["band_graphs"] and got["second"].meta["band_graphs"] == warm
    tiled._GRAPHS.clear()
