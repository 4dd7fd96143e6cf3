"""Tag reading with corners far outside the image: edges with more points than
are walked whole refine as the oracle's do, and edges of any finite length end,
without touching the quads beside them."""
import numpy as np
import pytest

from decode_ref import decode_one

from atag import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LAYOUT = synth.quadrant_layout(6)
CODES = synth.random_family(LAYOUT, 24, seed=4)


def _decode(img, quads):
    from atag import decode
    return decode.to_numpy(decode.decode_quads(torch.from_numpy(img).cuda(), torch.from_numpy(quads).cuda(),
                                               decode.Family(LAYOUT, CODES)))


@pytest.mark.parametrize("length", [32000.0, 34000.0, 120000.0])
def test_long_edges_refine_as_the_oracles(length):
    img, tags = synth.family_frame(3, LAYOUT, CODES, n_tags=3, width=700, height=420)
    quads = []
    for k, c in tags[:2]:
        d = (c[1] - c[0]) / np.linalg.norm(c[1] - c[0]) * length
        quads.append(np.stack([c[0] - d, c[1] + d, c[2] + d, c[3] - d]))  # through the tag's two sides
    quads = np.stack(quads).astype(np.float32)
    g = _decode(img, quads)
    for i, q in enumerate(quads):
        o = decode_one(img, q, LAYOUT, CODES)
        assert int(g["status"][i]) == o["status"]
        # corners are far out: compare them by their size
        scale = np.abs(o["corners"]).max()
        assert np.abs(g["corners"][i] - o["corners"]).max() <= 1e-3 + 1e-6 * scale


def test_edges_of_any_finite_length_end():
    img, tags = synth.family_frame(3, LAYOUT, CODES, n_tags=3, width=700, height=420)
    good = np.stack([c for _, c in tags]).astype(np.float32)
    far = []
    for v in (1e6, 1e9, 1e12, 1e20, 3e38):
        for corner in range(4):
            q = good[corner % len(good)].copy()
            q[corner] += np.sign(q[corner] - q.mean(0)) * np.float32(v)
            far.append(q)
    g = _decode(img, np.concatenate([good, np.stack(far), good]))
    n = len(good)
    assert g[:n].tobytes() == g[-n:].tobytes()
    assert sorted(g["id"][:n]) == sorted(k for k, _ in tags)
