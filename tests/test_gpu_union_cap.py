"""A union-find iteration cap with room for a union's two walks and its retries
is not raised by unions that contend for long chains, call after call, and the
labels are complete."""
import numpy as np
import pytest

import oracle
from conftest import synth_frame
from test_gpu_border_union import comb, spiral

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

IMAGES = {"spiral": lambda: spiral(540, 960, 8), "wide_spiral": lambda: spiral(600, 1280, 24),
          "comb": lambda: comb(720, 1280, 4), "1080p": lambda: synth_frame("1080p", 3)}


@pytest.mark.parametrize("cap", [14, 0xFFFFFFFF])
@pytest.mark.parametrize("name", sorted(IMAGES))
def test_caps_with_room_are_not_raised(name, cap):
    from atag.detector import Detector
    img = IMAGES[name]()
    det = Detector(img.shape[1], img.shape[0], keep_intermediates=True)
    det.set_limits(uf_iteration_cap=cap)
    g = torch.from_numpy(img).cuda()
    for _ in range(100):
        det.enqueue([g])
        assert int(det.stats()[0]["status"]) == 0
    want, _ = oracle.segmentation(oracle.threshold(img)[0])
    assert np.array_equal(np.asarray(det.views(0)["labels"]).reshape(want.shape), want)
