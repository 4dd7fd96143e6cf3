"""The outputs of a stage call are tensors of their own: one that a caller keeps
does not keep the others' memory, and none overlaps another."""
import pytest

from conftest import synth_frame

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_each_output_has_its_own_storage():
    from atag import stages
    grey = torch.from_numpy(synth_frame("vga", 3)).cuda()
    thr = stages.threshold_image(grey)
    labels, sizes, _ = stages.image_segmentation(thr)
    points, keys = stages.find_boundaries(labels, sizes)
    out, counts = stages.cluster(points, keys, grey)
    n, nc = int(counts["n_cluster_points"]), int(counts["n_clusters"])
    found = stages.fit_lines(out["line_fit"], out["cluster_indices"], out["cluster_extents"], n, on_device=True)
    corners, extents, _ = stages.corner_peaks(found, out["cluster_extents"], nc, n)
    tensors = [*out.values(), corners, extents]
    assert all(t.untyped_storage().nbytes() <= t.numel() + 7 for t in tensors)
    assert len({t.untyped_storage().data_ptr() for t in tensors}) == len(tensors)
    assert all(t.data_ptr() % 256 == 0 for t in tensors)
    # the part that no record was written to is zero
    assert int(out["line_fit"][64 * n:].count_nonzero()) == 0
