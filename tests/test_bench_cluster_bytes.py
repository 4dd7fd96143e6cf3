"""The bench's byte formulas of the cluster stages follow what the kernels move:
the sorts write each point's line-fit inputs (8 bytes), the window-error pass
reads those and writes the prefix sums (64)."""
from test_bench_formulas import _bench, _stats


def test_cluster_stage_bytes():
    b = _bench()
    st = _stats(64)
    Pf, K = 64 * 124_372, 64 * 5_000
    own = b.stage_bytes(st, 64 * 1920 * 1080)
    assert own["cluster_sort"] == 28 * Pf and own["cluster_errors"] == 72 * Pf
    survey = b.survey_bytes(st)
    assert survey["cluster_sort"] == 80 * Pf
    assert survey["cluster_errors"] == (96 + 96 + 2) * Pf + 12 * K
