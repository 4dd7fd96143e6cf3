"""corner_peaks on clusters of every size class: the smallest, those on both
sides of a warp's limit (256 points), ones without corners, and many at once;
and many small clusters take about the time of as many points in large ones."""
import numpy as np
import pytest

from gpu_helpers import assert_same

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _clusters(counts, share, seed):
    from atag import records as R
    rng = np.random.default_rng(seed)
    counts = np.asarray(counts)
    ext = np.zeros(len(counts), R.CLUSTER_EXTENTS)
    ext["count"] = counts
    ext["start"][1:] = np.cumsum(counts)[:-1]
    n = int(counts.sum())
    found = np.zeros(n, R.CORNER)
    hit = rng.random(n) < share
    found["error"][hit] = rng.integers(1, 50, int(hit.sum())).astype(np.float32)  # with ties
    found["cluster_index"] = np.repeat(np.arange(len(counts)), counts).astype(np.uint16)
    found["line_fit_point_index"] = np.arange(n) - np.repeat(ext["start"], counts)
    return found, ext


def _expected(found, ext):
    out, extents = [], []
    at = 0
    for e in ext:
        seg = found[e["start"]:e["start"] + e["count"]]
        seg = seg[seg["error"] != 0]
        if len(seg):
            out.append(seg[np.argsort(-seg["error"], kind="stable")])
            extents.append((at, len(seg)))
            at += len(seg)
    return np.concatenate(out).astype(found.dtype), np.array(extents, np.uint32)


@pytest.mark.parametrize("counts,share", [
    ([24, 25, 31, 32, 33, 255, 256, 257, 258, 1023, 1025, 5000], 0.3),
    ([256, 257] * 400, 0.5),
    ([24] * 20000, 0.12),
    ([24, 4000, 40] * 150, 0.02),
    ([256], 1.0),
    ([300] * 3 + [24] * 9725 + [300] * 5, 0.2),  # a round of all warps, large ones in each
])
def test_corners_of_clusters_of_all_sizes(counts, share):
    from atag import records as R, stages
    found, ext = _clusters(counts, share, len(counts))
    want, extents = _expected(found, ext)
    corners, pe, (k, cp, status) = stages.corner_peaks(stages.to_device(found), stages.to_device(ext), len(ext), len(found))
    assert status == 0 and (k, cp) == (len(want), len(extents))
    assert_same(stages.to_host(corners, R.CORNER)[:k], want, "corners")
    got = stages.to_host(pe, R.PEAK_EXTENTS)[:cp]
    assert np.array_equal(np.stack([got["start"], got["count"]], 1), extents)


def test_small_clusters_are_not_slower_than_large_ones():
    """A CTA per cluster of 24 points took 8 times as long as the same points in
    clusters of 1,200; a warp reads three quarters of its lanes' worth."""
    from atag import stages
    times = {}
    for size in (24, 1200):
        found, ext = _clusters([size] * (1440000 // size), 0.12, 5)
        f, e = stages.to_device(found), stages.to_device(ext)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(12)]
        for i in range(12):
            ev[i].record()
            for _ in range(10):
                stages.corner_peaks(f, e, len(ext), len(found))
        torch.cuda.synchronize()
        times[size] = float(np.median([ev[i].elapsed_time(ev[i + 1]) for i in range(1, 11)]))
    assert times[24] <= 3 * times[1200], times
