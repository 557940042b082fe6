"""detect_centers of small frames with the counts left on the device (one wait) against the flow that reads them
first, exactly; frames with more components than there is room for, and the label prefix in one launch against
the three-launch form's numbering (the oracle's labels) on either side of its size limit."""

import numpy as np
import pytest

from oracle import segment as osg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("refine", ["auto", "logquad", "weighted", "none", "edge_moment"])
def test_matches_the_counted_flow(dtype, refine):
    from imageprocessor_new_b200 import _device as dev, centers, segment, synthetic

    page = synthetic.page_square(2, shape=(200, 333)).image
    img = (page >> 4).astype(dtype) if np.dtype(dtype) == np.uint8 else page.astype(dtype)
    for crop, morph in ((img, 0), (np.ascontiguousarray(img[:7, :9]), 0), (np.ascontiguousarray(img[50:131, 3:260]), 1)):
        d = dev.upload(crop)
        common = dict(threshold_dev=segment.otsu(dev.upload(page[:crop.shape[0], :crop.shape[1]])) if dtype == np.float32
                      else segment.otsu(d), fixed_threshold=0.0, invert=False, area_min=2, area_max=400, pad=3,
                      refine=refine, connectivity=8, small_feature_max=12.0, morph_open=morph, morph_close=morph)
        got = centers._centers_in_one_wait(d, **common)
        want = centers._finite(centers._centers_on_device(d, **common))
        np.testing.assert_array_equal(got, want)


def test_more_components_than_room():
    from imageprocessor_new_b200 import _device as dev, centers, detect_centers

    img = np.zeros((64, 128), np.uint8)
    img[::3, ::3] = 200  # a component in every nine pixels
    d = dev.upload(img)
    common = dict(threshold_dev=None, fixed_threshold=100.0, invert=False, area_min=1, area_max=9, pad=1,
                  refine="weighted", connectivity=8, small_feature_max=12.0)
    assert centers._centers_in_one_wait(d, **common) is None
    want = centers._finite(centers._centers_on_device(d, **common))
    res = detect_centers(img, threshold="otsu", area_min=1, area_max=9, pad=1, refine="weighted", backend="gpu")
    np.testing.assert_array_equal(res.centers_xy, want)
    assert len(want) == 22 * 43


@pytest.mark.parametrize("shape", [(64, 64), (127, 1031), (2048, 2112), (2049, 2113), (2113, 2200)])
def test_label_prefix_around_its_limit(shape):
    from imageprocessor_new_b200 import segment

    rng = np.random.default_rng(shape[1])
    fg = rng.random(shape) < 0.2
    res = segment.connected_components_stats(fg.astype(np.uint8), connectivity=8)
    num, labels, stats, _ = osg.label_components(fg, 8)
    assert res.num_labels == num
    np.testing.assert_array_equal(res.labels, labels)
    np.testing.assert_array_equal(res.stats[1:], stats[1:])
