"""A frame's pair table that is nearly or completely full: keys placed by the
merge count the same points as in a table with room, and every slot is used
before a pair is dropped."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _squares(height, width, pitch, size, tilt):
    yy, xx = np.mgrid[0:height, 0:width]
    u, v = np.cos(tilt) * xx + np.sin(tilt) * yy, np.cos(tilt) * yy - np.sin(tilt) * xx
    img = np.full((height, width), 230, np.uint8)
    img[((u % pitch) < size) & ((v % pitch) < size)] = 20
    return img


def _pairs(view):
    keys = view["pair_keys"]
    used = keys != np.uint64(0xFFFFFFFFFFFFFFFF)
    rows = np.concatenate([view["pair_count"][used, None].astype(np.int64), view["pair_bbox"][used].astype(np.int64),
                           view["pair_gsum"][used].astype(np.int64), view["pair_pxgx"][used, None]], 1)
    return dict(zip(keys[used].tolist(), map(tuple, rows.tolist())))


@pytest.mark.parametrize("tilt", [0.0, 0.3])
def test_pairs_of_a_full_table(tilt):
    from atag import records as R
    from atag.detector import Detector
    img = torch.from_numpy(_squares(600, 800, 40, 24, tilt)).cuda()
    det = Detector(800, 600, keep_intermediates=True)
    _, st = det.detect([img])
    whole = _pairs(det.views(0))
    assert int(st[0]["status"]) == 0 and len(whole) > 256
    room = 1 << (len(whole) - 1).bit_length()
    for capacity in (room, room // 2, 64, 2):
        det.set_limits(pair_capacity=capacity)
        for _ in range(3):
            _, st = det.detect([img])
            got = _pairs(det.views(0))
            if capacity >= len(whole):
                assert int(st[0]["status"]) == 0 and got == whole
                continue
            assert int(st[0]["status"]) & R.DEVFLAG_PAIR_OVERFLOW
            assert len(got) == int(st[0]["n_pairs"]) == capacity
            assert all(whole[k] == v for k, v in got.items())
