"""The points of tag reading's edge refinement on edges of any length: none
that can meet the image is left out, and their number is bounded by the image
(compiled for the host from the device's header)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not installed")
def test_points_that_can_meet_the_image(tmp_path):
    exe = tmp_path / "edge_samples_check"
    subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "native", "edge_samples_check.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout
    edges, bad = map(int, out.stdout.split()[-2:])
    assert edges > 5000 and bad == 0
