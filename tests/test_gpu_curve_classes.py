"""Curve flattening with one to 32 lanes per curve against the oracle, byte
for byte: curves of every length class (from one leaf to thousands), alone and
so many that each gets fewer lanes, curves that return to their start (their
edges are not their leaves' chords), degenerate ones, and the stroker's
subdivision of a few and of many nodes."""
import numpy as np
import pytest

from backends import GpuBackend, StrokeOracle
from z2d_gb300 import abi, painter
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import FillOptions, Pattern, Pixel, StrokeOptions

pytestmark = pytest.mark.gpu
W, H = 160, 90
PIX = Pattern.from_pixel(Pixel.rgba(150, 60, 10, 200))


@pytest.fixture(scope="module")
def gpu():
    return GpuBackend()


def _curves(rng, n, size, shape):
    p = Path()
    x, y = rng.uniform(0, W), rng.uniform(0, H)
    p.move_to(x, y)
    for k in range(n):
        a = rng.uniform(-size, size, 6)
        if shape == "loop":  # ends, and passes its middle, where it started
            p.curve_to(x + a[0], y + a[1], x - a[0], y - a[1], x, y)
        elif shape == "flat":  # control points on the chord, some equal
            q = (x + a[4], y + a[5])
            p.curve_to(x, y, *(q if k % 2 else (x + a[4] / 2, y + a[5] / 2)), *q)
            x, y = q
        else:
            x1, y1 = min(max(x + a[4], -W), 2 * W), min(max(y + a[5], -H), 2 * H)
            p.curve_to(x + a[0], y + a[1], x + a[2], y + a[3], x1, y1)
            x, y = x1, y1
    p.line_to(rng.uniform(0, W), rng.uniform(0, H))
    p.close()
    return p.to_array()


def _off_surface():
    p = Path()
    p.move_to(-5000, -5000)
    for k in range(4200):
        p.line_to(-4000 - (k % 7), -5000 + k * 0.01)
    p.close()
    return p.to_array()


@pytest.mark.parametrize("size", [0.05, 0.5, 3.0, 12.0, 50.0, 200.0, 900.0, 6000.0])
@pytest.mark.parametrize("n", [1, 5, 33])
@pytest.mark.parametrize("shape", ["free", "loop", "flat"])
def test_classes(gpu, oracle, size, n, shape):
    rng = np.random.default_rng(int(size * 100) + n)
    for tol in (0.1, 0.004):
        nodes, opts = _curves(rng, n, size, shape), FillOptions(tolerance=tol)
        a, b = Surface.init("rgba", W, H), Surface.init("rgba", W, H)
        painter.fill_batch(a, [(PIX, nodes, opts), (PIX, _off_surface(), opts)], ctx=gpu.ctx)
        assert oracle.fill(b, PIX, nodes, opts) == abi.OK
        assert np.array_equal(a.numpy(), b.numpy()), (size, n, shape, tol)


def test_many_curves_of_all_classes(gpu, oracle):
    """More curves than the grid has lanes: one lane each for the short ones."""
    rng = np.random.default_rng(3)
    fills = [(PIX, _curves(rng, 3000, float(s), "free"), FillOptions(fill_rule="even_odd"))
             for s in [1.0] * 20 + [8.0] * 8 + [40.0] * 4 + [150.0]]
    a, b = Surface.init("rgba", W, H), Surface.init("rgba", W, H)
    painter.fill_batch(a, fills, ctx=gpu.ctx)
    for f in fills:
        assert oracle.fill(b, *f) == abi.OK
    assert np.array_equal(a.numpy(), b.numpy())


@pytest.mark.parametrize("size", [0.5, 30.0, 900.0])
@pytest.mark.parametrize("n", [1, 7, 12000])
def test_strokes(gpu, oracle, size, n):
    rng = np.random.default_rng(n)
    if n > 1000:
        size = min(size, 30.0)
    nodes = _curves(rng, n, size, "free")
    opts = StrokeOptions(line_width=3.0, line_join="round")
    a, b = Surface.init("rgba", W, H), Surface.init("rgba", W, H)
    rc = gpu.stroke(a, PIX, nodes, opts)
    assert rc == StrokeOracle(oracle).stroke(b, PIX, nodes, opts)
    assert np.array_equal(a.numpy(), b.numpy())
