"""Kernels whose CTAs are placed while the previous kernel runs, on inputs that
change from call to call: every pass over frames of the same sizes and other
contents, some of them nearly empty, gives the quads and counts that kernels
launched one after the other give (a detector that records stage events does
not place them early).  Data left by the pass before would show."""
import numpy as np
import pytest

from conftest import synth_frame

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _square(height, width):
    img = np.full((height, width), 200, np.uint8)
    img[100:180, 120:200] = 30
    return img


def _lists(names, colour):
    """Contents 0 and 1: rendered frames; 2: one square each; 3: flat."""
    out = []
    for content in range(4):
        frames = []
        for k, name in enumerate(names):
            img = synth_frame(name, 10 + 7 * content + k)
            if content == 2:
                img = _square(*img.shape)
            if content == 3:
                img = np.full_like(img, 128)
            t = torch.from_numpy(img).cuda()
            frames.append(t[..., None].expand(-1, -1, 3).contiguous() if colour else t)
        out.append(frames)
    return out


@pytest.mark.parametrize("names,lanes,colour,refine", [
    (["1080p"], 1, False, False), (["vga"], 1, True, True), (["vga", "1080p", "vga"], 1, False, True),
    (["1080p", "vga", "vga", "1080p"], 2, False, False), (["vga"] * 7, 4, True, True)])
def test_every_pass_is_its_own(names, lanes, colour, refine):
    from atag import lib
    from atag.detector import Detector
    lists = _lists(names, colour)
    n = len(names)

    def detector():
        det = Detector(1920, 1080, max_frames=n)
        det.set_refinement(refine)
        return det

    plain = detector()
    plain.set_stage_events([torch.cuda.Event(enable_timing=True) for _ in range(lib.STAGE_COUNT + 1)])
    want, counts = [], []
    for frames in lists:
        quads, stats = plain.detect(frames)
        want.append([q.tobytes() for q in quads])
        counts.append(stats.copy())
    assert sum(len(q) for q in want[0]) > 0 and want[0] != want[1]
    assert all(len(q) == 0 for q in want[3])

    det = detector()
    det.set_tuning(batch_lanes=lanes)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    order = [0, 3, 1, 2, 0, 1, 3, 2, 2, 0] * 4
    passes = []
    for which in order:
        det.enqueue(lists[which], stream=stream)
        with torch.cuda.stream(stream):
            passes.append((det.d_quads.clone(), det.d_stats.clone()))
    stream.synchronize()
    for which, (d_quads, d_stats) in zip(order, passes):
        det.d_quads, det.d_stats = d_quads, d_stats
        quads, stats = det.results()
        assert [q.tobytes() for q in quads] == want[which]
        assert stats.tobytes() == counts[which].tobytes()
