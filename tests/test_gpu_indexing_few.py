"""do_indexing does not read the corners of clusters with fewer than four, which
make no quad: extents past the end of a truncated corner array stay unread."""
import numpy as np
import pytest

import oracle
from conftest import synth_frame

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


def test_extents_of_few_corners_past_the_array():
    from atag import stages
    res = oracle.detect(synth_frame("1080p", 2))
    pe = res["peak_extents"].copy()
    few = np.arange(len(pe)) % 3 == 0
    pe["start"][few] = 1 << 30
    pe["count"][few] = 1 + np.arange(int(few.sum())) % 3
    # cluster extents by the peak extents' position, as the reference reads them
    got = stages.do_indexing(pe, res["corners"], res["line_fit"], res["extents"][:len(pe)])
    ref = oracle.do_indexing(res["peak_extents"], res["corners"], res["line_fit"], res["extents"][:len(pe)])
    ref[few] = np.zeros(1, ref.dtype)
    assert np.array_equal(got, ref)
