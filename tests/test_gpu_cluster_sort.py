"""The cluster sort where its buckets are uneven or its storage changes: long
thin shapes (most keys in the buckets next to an axis), large round ones (many
equal thetas), clusters on both sides of the small/large split, and clusters
past the shared-memory capacity (frames larger than 3840 x 2160)."""
import numpy as np
import pytest

import oracle
from gpu_helpers import assert_detect_matches

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def frame(width, height, shapes):
    """Black shapes on white: ("disk", cx, cy, r) or ("bar", cx, cy, half
    length, half width, angle)."""
    yy, xx = np.mgrid[0:height, 0:width].astype(np.float32)
    img = np.full((height, width), 255, np.uint8)
    for s in shapes:
        if s[0] == "disk":
            img[(xx - s[1]) ** 2 + (yy - s[2]) ** 2 <= s[3] ** 2] = 0
        else:
            _, cx, cy, a, b, t = s
            u, v = np.cos(t) * (xx - cx) + np.sin(t) * (yy - cy), np.cos(t) * (yy - cy) - np.sin(t) * (xx - cx)
            img[(np.abs(u) <= a) & (np.abs(v) <= b)] = 0
    return img


CASES = {
    # bars along the axes, the diagonal and just off an axis
    "thin": (1284, 964, [("bar", 640, 60, 600, 1.2, 0.0), ("bar", 60, 500, 1.2, 400, 0.0),
                         ("bar", 600, 500, 380, 1.6, 0.7854), ("bar", 700, 150, 500, 2.0, 0.004)]),
    "small": (324, 244, [("disk", 40, 40, 4), ("disk", 120, 60, 20), ("disk", 220, 130, 55)]),
    "split": (1924, 1084, [("disk", 240, 240, 126), ("disk", 700, 240, 130), ("disk", 1500, 500, 400)]),
    "beyond_shared": (4096, 2400, [("bar", 2048, 1200, 1900, 1190, 0.0)]),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_sorted_points_and_prefix_sums(name):
    from atag.detector import Detector
    w, h, shapes = CASES[name]
    img = frame(w, h, shapes)
    det = Detector(w, h, keep_intermediates=True)
    quads, _ = det.detect([torch.from_numpy(img).cuda()])
    res = oracle.detect(img)
    counts = res["extents"]["count"]
    assert len(counts) == len(shapes)
    if name == "split":
        assert (counts <= 2048).any() and ((counts > 2048) & (counts < 2200)).any()
    if name == "beyond_shared":
        assert counts.max() > 24576
    assert_detect_matches(det.views(0), quads[0], res)


def test_any_split_sorts_the_same():
    from atag.detector import Detector
    img = frame(*CASES["split"])
    g = torch.from_numpy(img).cuda()
    det = Detector(img.shape[1], img.shape[0])
    det.detect([g])
    want = det.views(0)
    for split in (1, 37, 256, 257, 2047):
        det.set_tuning(small_cluster_max=split)
        det.detect([g])
        got = det.views(0)
        for k in ("cluster_points", "line_fit", "peaks", "fitted"):
            assert got[k].tobytes() == want[k].tobytes(), (split, k)
