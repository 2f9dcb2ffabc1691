"""Edges that reach beyond 2^31 sample rows: the bins' records on the host
(tests/bin_edge_range_check.cu, built with nvcc as host code and the undefined
behaviour sanitizer), and strokes of such widths on the GPU."""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_records_at_the_ends_of_the_range():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "bin_edge_range_check")
        subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17",
                        "-Xcompiler", "-ffp-contract=off,-fsanitize=undefined,-fno-sanitize-recover=undefined",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "z2d_gb300", "csrc"),
                        os.path.join(HERE, "bin_edge_range_check.cu"), "-o", exe, "-lubsan"], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "wrong 0" in r.stdout, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("width", [1.0e9, 1.5e9, 3.0e9])
@pytest.mark.parametrize("aa", ["default", "none"])
def test_stroke_beyond_the_range(width, aa):
    """A horizontal line so wide that its outline's upright edges begin and end
    beyond the sample rows' range: its columns, on every row."""
    from z2d_gb300 import painter
    from z2d_gb300.path import Path
    from z2d_gb300.surface import Surface
    from z2d_gb300.types import Pattern, Pixel, StrokeOptions
    s = Surface.init("rgba", 120, 70)
    painter.stroke(s, Pattern.from_pixel(Pixel.rgba(10, 20, 30, 255)), Path().move_to(10, 35).line_to(100, 35).to_array(),
                   StrokeOptions(line_width=width, anti_aliasing=aa))
    want = np.zeros((70, 120, 4), np.uint8)
    want[:, 10:100] = (10, 20, 30, 255)
    assert np.array_equal(s.pixels(), want)
