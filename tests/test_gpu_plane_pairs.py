"""atag_cluster's pass over the dense planes: one pair of nearly all points
(long runs of one key), more pairs in a stretch than the block's table holds,
random ternary-like noise (a key per few entries), and frames smaller than one
group of entries; and the corner peaks of clusters of any size."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def image(name):
    rng = np.random.default_rng(5)
    if name == "noise":
        return rng.integers(0, 256, (240, 320), dtype=np.uint8)
    if name == "tiny":
        return np.kron(rng.integers(0, 2, (4, 5), dtype=np.uint8) * 255, np.ones((4, 4), np.uint8))
    if name == "one_pair":
        img = np.full((400, 1280), 255, np.uint8)
        img[4:396:8, 4:1276] = 0
        img[4:396, 636:644] = 0
        return img
    if name == "blobs":
        img = np.full((480, 640), 255, np.uint8)
        for k, r in enumerate((6, 9, 14, 20, 27, 35, 44, 54)):
            yy, xx = np.mgrid[0:480, 0:640]
            img[(xx - 80 - 160 * (k % 4)) ** 2 + (yy - 120 - 240 * (k // 4)) ** 2 <= r * r] = 0
        return img
    img = np.zeros((600, 1920), np.uint8)  # 119 squares to a row; the frame's table holds 4096 pairs
    for k in range(119 * 18):
        y, x = divmod(k, 119)
        img[4 + 16 * y:13 + 16 * y, 4 + 16 * x:13 + 16 * x] = 255
    return img


@pytest.mark.parametrize("name", ["noise", "tiny", "one_pair", "blobs", "squares"])
def test_pairs_clusters_and_peaks(name):
    from atag import records as R
    from atag import stages
    img = image(name)
    h, w = img.shape
    res = oracle.detect(img)
    grey = torch.from_numpy(img).cuda()
    labels, sizes, _ = stages.image_segmentation(stages.threshold_image(grey))
    out, counts = stages.cluster(*stages.find_boundaries(labels, sizes), grey)
    assert int(counts["status"]) == 0
    C, n, nc = int(counts["n_pairs"]), int(counts["n_cluster_points"]), int(counts["n_clusters"])
    assert (C, n, nc) == (len(res["bounds"]), len(res["cluster_points"]), len(res["extents"]))
    assert stages.to_host(out["pair_bounds"], R.CLUSTER_BOUNDS)[:C].tobytes() == res["bounds"].tobytes()
    assert stages.to_host(out["cluster_points"], R.CLUSTER_POINT)[:n].tobytes() == res["cluster_points"].tobytes()
    assert stages.to_host(out["line_fit"], R.LINE_FIT_POINT)[:n].tobytes() == res["line_fit"].tobytes()
    if nc == 0:
        return
    found = stages.fit_lines(out["line_fit"], out["cluster_indices"], out["cluster_extents"], n, on_device=True)
    corners, pe, (k, cp, status) = stages.corner_peaks(found, out["cluster_extents"], nc, n)
    assert (k, cp, status) == (len(res["corners"]), len(res["peak_extents"]), 0)
    assert np.array_equal(np.sort(stages.to_host(corners, R.CORNER)[:k]["error"]), np.sort(res["corners"]["error"]))
    assert stages.to_host(pe, R.PEAK_EXTENTS)[:cp].tobytes() == res["peak_extents"].tobytes()
