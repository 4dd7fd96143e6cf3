"""The key sort of the pair finalisation at the sizes where its form changes:
one, two and four keys a thread, shared memory by the whole CTA, and in place
in global memory; and several frames of different counts in one batch, whose
work lists the last frame's CTA makes."""
import numpy as np
import pytest

import oracle
from gpu_helpers import assert_detect_matches

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def squares(count):
    """count white squares (pairs whose blobs the filter drops: only dark on
    white passes), a white margin (a pair more) with a dark bar on it (another,
    which stays)."""
    img = np.zeros((1096, 1920), np.uint8)
    for k in range(count):
        y, x = divmod(k, 119)
        img[4 + 16 * y:13 + 16 * y, 4 + 16 * x:13 + 16 * x] = 255
    img[:, -16:] = 255
    img[300:360, -12:-2] = 0
    return img


@pytest.mark.parametrize("pairs", [3, 33, 1024, 1025, 2048, 2049, 4096, 4097, 6048, 6049, 7900])
def test_any_number_of_pairs(pairs):
    from atag.detector import Detector
    img = squares(pairs - 2)
    res = oracle.detect(img)
    assert len(res["bounds"]) == pairs and len(res["extents"]) == 1
    det = Detector(1920, 1096, keep_intermediates=True)
    quads, _ = det.detect([torch.from_numpy(img).cuda()])
    assert_detect_matches(det.views(0), quads[0], res)


@pytest.mark.parametrize("frames", [2, 33, 65])
def test_lists_of_a_batch(frames):
    from atag.detector import Detector
    counts = [0, 5, 700, 40]
    imgs = [torch.from_numpy(np.ascontiguousarray(squares(c)[:600])).cuda() for c in counts]
    alone = Detector(1920, 600)
    want = []
    for g in imgs:
        q, st = alone.detect([g])
        want.append((q[0].tobytes(), st[0].tobytes()))
    det = Detector(1920, 600, max_frames=frames)
    det.set_tuning(batch_lanes=1)
    q, st = det.detect([imgs[k % 4] for k in range(frames)])
    for k in range(frames):
        assert (q[k].tobytes(), st[k].tobytes()) == want[k % 4], k
