"""Kernels whose CTAs are placed while the previous kernel runs: lanes on both
sides of the pixel limit, one and several lanes, launched and replayed, many
times in a row on one detector, give the results of each frame alone."""
import numpy as np
import pytest

from conftest import synth_frame

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("frames,lanes", [(1, 1), (3, 2), (4, 2), (8, 2), (7, 4), (5, 1)])
def test_results_do_not_depend_on_the_launch(frames, lanes):
    from atag.detector import Detector
    images = [torch.from_numpy(synth_frame("1080p" if k % 3 else "vga", k)).cuda() for k in range(frames)]
    alone = Detector(1920, 1080)
    want = []
    for f in images:
        q, st = alone.detect([f])
        want.append(q[0].tobytes())
        assert len(q[0]) > 0
    det = Detector(1920, 1080, max_frames=frames)
    det.set_tuning(batch_lanes=lanes)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def check():
        stream.synchronize()
        got, st = det.results()
        assert [q.tobytes() for q in got] == want

    for _ in range(20):
        det.enqueue(images, stream=stream)
    check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        det.enqueue(images, stream=stream)
    with torch.cuda.stream(stream):
        for _ in range(20):
            graph.replay()
    check()
