"""The combination search and the corner intersection on chosen inputs: every
number of peaks around the sizes of the segment table, peaks in any order of
position, and quad counts around the groups of the ordered compaction."""
import numpy as np
import pytest

import oracle
from conftest import synth_frame
from gpu_helpers import assert_quads_match

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def clusters():
    return oracle.detect(synth_frame("1080p", 2))


@pytest.mark.parametrize("peaks", [3, 4, 5, 9, 10, 11, 40])
def test_any_peaks_in_any_order(clusters, peaks):
    """Fitted quads are whole numbers and equal the oracle's."""
    from atag import stages
    rng = np.random.default_rng(peaks)
    ext = clusters["extents"]
    ext = ext[ext["count"] > 2 * peaks]
    assert len(ext) > 20
    corners = np.zeros(len(ext) * peaks, clusters["corners"].dtype)
    pe = np.zeros(len(ext), clusters["peak_extents"].dtype)
    for q, e in enumerate(ext):
        corners["line_fit_point_index"][q * peaks:(q + 1) * peaks] = 1 + rng.choice(int(e["count"]) - 2, peaks, replace=False)
        if q % 3 == 0:  # the very first and last point of the cluster
            corners["line_fit_point_index"][q * peaks:q * peaks + 2] = (e["count"] - 1, 0)
        corners["cluster_index"][q * peaks:(q + 1) * peaks] = q
        pe[q] = (q * peaks, peaks)
    got = stages.do_indexing(pe, corners, clusters["line_fit"], ext)
    want = oracle.do_indexing(pe, corners, clusters["line_fit"], ext)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("count", [1, 127, 128, 129, 400])
def test_quads_in_order(clusters, count):
    """Eight lanes per quad, 128 quads per round of the compaction."""
    from atag import stages
    rng = np.random.default_rng(count)
    fitted = np.ascontiguousarray(rng.choice(clusters["fitted"], count))
    got = stages.process_fitted_quads(fitted, clusters["width"], clusters["height"])
    want = oracle.process_fitted_quads(fitted)
    assert_quads_match(got, want)
