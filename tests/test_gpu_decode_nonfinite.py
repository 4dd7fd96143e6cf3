"""Quads with a corner that is not finite are degenerate: no pixel is read at
their projections, with and without edge refinement, and the quads beside them
decode as they do alone."""
import itertools

import numpy as np
import pytest

from decode_ref import DEGENERATE, REORDERED, decode_one

from atag import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LAYOUT = synth.quadrant_layout(6)
CODES = synth.random_family(LAYOUT, 24, seed=4)


@pytest.mark.parametrize("refine", [0, 1])
def test_corners_that_are_not_finite(refine):
    from atag import decode
    img, tags = synth.family_frame(3, LAYOUT, CODES, n_tags=3, width=700, height=420)
    good = np.stack([c for _, c in tags]).astype(np.float32)
    bad = []
    for corner, axis, value in itertools.product(range(4), range(2), (np.inf, -np.inf, np.nan)):
        q = good[corner % len(good)].copy()
        q[corner, axis] = value
        bad += [q, q[[0, 3, 2, 1]]]
    quads = np.concatenate([good, np.stack(bad), good])
    prm = decode.default_params(refine_edges=refine)
    fam = decode.Family(LAYOUT, CODES)
    g = decode.to_numpy(decode.decode_quads(torch.from_numpy(img).cuda(), torch.from_numpy(quads).cuda(), fam, prm))
    n = len(good)
    assert ((g["status"][n:-n] & ~np.uint32(REORDERED)) == DEGENERATE).all()
    assert (g["id"][n:-n] == -1).all()
    assert g[:n].tobytes() == g[-n:].tobytes()
    assert sorted(g["id"][:n]) == sorted(k for k, _ in tags)
    with np.errstate(invalid="ignore"):
        assert all(decode_one(img, q, LAYOUT, CODES, refine=bool(refine))["status"] & DEGENERATE for q in bad)
