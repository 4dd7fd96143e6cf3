"""Unions across tile borders on components that run through many tiles and
meet late: spirals and combs, whole and cut, through the stage entry point
and the detector's path."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def spiral(height, width, step):
    """A white line, step / 2 wide, winding inwards on black."""
    img = np.zeros((height, width), np.uint8)
    t, l, b, r = 0, 0, height, width
    while b - t > 2 * step and r - l > 2 * step:
        img[t:t + step // 2, l:r] = 255
        img[t:b, r - step // 2:r] = 255
        img[b - step // 2:b, l + step:r] = 255
        img[t + step:b, l + step:l + step + step // 2] = 255
        t, l, b, r = t + step, l + step, b - step, r - step
    return img


def comb(height, width, step):
    img = np.zeros((height, width), np.uint8)
    img[:, ::step] = 255
    img[:, 1::step] = 255
    img[-2:] = 255
    return img


IMAGES = {"spiral": lambda: spiral(540, 960, 8), "wide_spiral": lambda: spiral(600, 1280, 24),
          "comb": lambda: comb(360, 1280, 4), "rows": lambda: np.ascontiguousarray(comb(1280, 360, 4).T)}


@pytest.mark.parametrize("name", sorted(IMAGES))
def test_stage_labels(name):
    from atag import stages
    thr = IMAGES[name]()
    labels, sizes, _ = stages.image_segmentation(torch.from_numpy(thr).cuda())
    want, want_sizes = oracle.segmentation(thr)
    assert np.array_equal(labels.cpu().numpy().view(np.uint32), want)
    assert np.array_equal(sizes.cpu().numpy().view(np.uint32), want_sizes)


@pytest.mark.parametrize("rows", [8, 16, 32])
@pytest.mark.parametrize("name", sorted(IMAGES))
def test_detector_labels(name, rows):
    from atag.detector import Detector
    img = IMAGES[name]()
    det = Detector(img.shape[1], img.shape[0], keep_intermediates=True)
    det.set_tuning(ccl_tile_rows=rows)
    det.detect([torch.from_numpy(img).cuda()])
    want, want_sizes = oracle.segmentation(oracle.threshold(img)[0])
    v = det.views(0)
    assert np.array_equal(np.asarray(v["labels"]).reshape(want.shape), want)
    assert np.array_equal(np.asarray(v["sizes"]).reshape(want_sizes.shape), want_sizes)
