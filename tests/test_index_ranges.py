"""Index arithmetic at the sizes where 32 bits end: on the host
(tests/index_check.cu, built with nvcc as host code), and batches of more
than 2^27 four-row bands on the GPU."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_item_numbers():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "index_check")
        subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "z2d_gb300", "csrc"),
                        os.path.join(HERE, "index_check.cu"), "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_more_than_2_27_bands():
    """66 surfaces of one column and 2^23 - 1 rows, each filled from top to
    bottom: 66 * 2^21 bands of one fill."""
    torch = pytest.importorskip("torch")
    from z2d_gb300 import painter
    from z2d_gb300.native import Context
    from z2d_gb300.path import Path
    from z2d_gb300.surface import Surface
    from z2d_gb300.types import FillOptions, Pattern, Pixel
    if torch.cuda.mem_get_info()[0] < 32 << 30:
        pytest.skip("needs 32 GB of device memory")
    h = (1 << 23) - 1
    nodes = Path().move_to(0, 0).line_to(1, 0).line_to(1, h).line_to(0, h).close().to_array()
    pat = Pattern.from_pixel(Pixel.rgba(0, 0, 0, 200))
    dev = [Surface.init("alpha8", 1, h).to_device("cuda") for _ in range(66)]
    torch.cuda.synchronize()
    ctx = Context(0)
    painter.fill_jobs([(d, [(pat, nodes, FillOptions())]) for d in dev], ctx=ctx)
    ctx.synchronize()
    ctx.close()
    for k, d in enumerate(dev):
        other = int((d.data != 200).sum())
        assert other == 0, f"surface {k}"


@pytest.mark.gpu
def test_layer_of_the_widest_row():
    """A row of 2^31 - 1 alpha8 pixels composited onto another."""
    torch = pytest.importorskip("torch")
    from z2d_gb300 import compositor
    from z2d_gb300.surface import Surface
    w = (1 << 31) - 1
    if torch.cuda.mem_get_info()[0] < 16 << 30:
        pytest.skip("needs 16 GB of device memory")
    src = torch.full((w,), 60, dtype=torch.uint8, device="cuda")
    src[-3:] = 200
    dst = torch.full((w,), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    compositor.composite(Surface("alpha8", w, 1, dst), Surface("alpha8", w, 1, src), "dst_in", 0, 0)
    torch.cuda.synchronize()
    same = torch.equal(dst, src)  # 255 * s / 255
    assert same


@pytest.mark.gpu
def test_gradient_on_the_widest_rows():
    """A gradient through a mask onto two rows of 2^31 - 1 alpha8 pixels: beyond
    its end every pixel of both rows has the last stop's alpha."""
    torch = pytest.importorskip("torch")
    from z2d_gb300 import compositor
    from z2d_gb300.surface import Surface
    from z2d_gb300.types import Color, Gradient, Operation, Pattern
    w, end = (1 << 31) - 1, 1 << 20
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    mask = torch.full((2 * w,), 255, dtype=torch.uint8, device="cuda")
    dst = torch.zeros(2 * w, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    g = Gradient.linear(0, 0, end, 0)
    g.add_stop(0.0, Color.rgb(0, 0, 0, 0)).add_stop(1.0, Color.rgb(0, 0, 0, 1))
    compositor.SurfaceCompositor.run(Surface("alpha8", w, 2, dst), 0, 0,
                                     [Operation("dst_in", dst=Pattern.from_gradient(g), src=Surface("alpha8", w, 2, mask)),
                                      Operation("src")])
    torch.cuda.synchronize()
    for y in (0, 1):
        row = dst[y * w:(y + 1) * w]
        first, other = int(row[0]), int((row[end:] != 255).sum())
        assert first == 0 and other == 0, f"row {y}"
