"""Edge refinement of the tag reader against the oracle where its walk along
the normals changes: search ranges from one to eight pixels, corners past the
limit of the integer positions (4,000 px), and corners next to and outside
the image's sides."""
import numpy as np
import pytest

from decode_ref import decode_one

from atag import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LAYOUT = synth.quadrant_layout(6)
CODES = synth.random_family(LAYOUT, 24, seed=4)


def _compare(img, quads, quad_decimate):
    from atag import decode
    fam = decode.Family(LAYOUT, CODES)
    prm = decode.default_params(quad_decimate=quad_decimate)
    g = decode.to_numpy(decode.decode_quads(torch.from_numpy(img).cuda(), torch.from_numpy(quads).cuda(), fam, prm))
    for i, q in enumerate(quads):
        o = decode_one(img, q, LAYOUT, CODES, quad_decimate=quad_decimate)
        assert int(g["status"][i]) == o["status"], i
        assert np.abs(g["corners"][i] - o["corners"]).max() < 1e-3, i
        if o["status"] & 2:
            continue
        assert abs(float(g["black"][i]) - o["black"]) < 1e-3 and abs(float(g["white"][i]) - o["white"]) < 1e-3
        assert abs(float(g["decision_margin"][i]) - o["decision_margin"]) < 1e-3
        assert int(g["code"][i]) == o["code"] and int(g["id"][i]) == o["id"]
        assert int(g["hamming"][i]) == o["hamming"] and int(g["rotation"][i]) == o["rotation"]


@pytest.mark.parametrize("width", [700, 4700])
@pytest.mark.parametrize("quad_decimate", [1, 3, 8])
def test_refined_quads_equal_the_oracles(width, quad_decimate):
    img, tags = synth.family_frame(width + quad_decimate, LAYOUT, CODES, n_tags=6, width=width, height=420)
    rng = np.random.default_rng(width)
    quads = np.stack([c for _, c in tags]) + rng.uniform(-0.7, 0.7, (len(tags), 4, 2))
    if width > 4000:  # and quads across the limit
        quads = np.concatenate([quads, quads[:2] - quads[:2].mean(1, keepdims=True) + [[[4000.0, 200.0]]]])
    _compare(img, quads.astype(np.float32), quad_decimate)


def test_corners_at_and_outside_the_sides():
    img, tags = synth.family_frame(3, LAYOUT, CODES, n_tags=3, width=700, height=420)
    c = tags[0][1]
    quads = np.stack([c - c.mean(0) + [20.3, 210.2], c - c.mean(0) + [680.7, 11.1], c,
                      c - c.min(0) + 0.25, c - c.max(0) + [699.2, 419.3]])
    quads[2] = quads[2][[0, 3, 2, 1]]
    _compare(img, quads.astype(np.float32), 1)
