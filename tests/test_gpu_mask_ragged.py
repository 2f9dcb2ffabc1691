"""Whole-surface mask batches whose pixel count is no whole number of the
kernels' 16-byte chunks, gradient sources on the alpha formats and alpha8 layers, against
the oracle: the smallest surfaces (a tail alone), chunk edges, and more than
one block."""
import numpy as np
import pytest

from backends import GpuBackend
from z2d_gb300 import abi
from z2d_gb300.surface import Surface
from z2d_gb300.types import Color, Gradient, Operation, Pattern, Pixel

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (3, 1), (5, 1), (15, 1), (17, 1), (33, 3), (31, 31), (257, 17), (1573, 11)]


@pytest.fixture(scope="module")
def gpu():
    return GpuBackend()


def _check(gpu, oracle, fmt, w, h, src, op, precision):
    rng = np.random.default_rng(w + 31 * h)
    mask = Surface.init("alpha8", w, h)
    mask.data[:] = rng.integers(0, 256, mask.data.size, dtype=np.uint8)
    a, b = Surface.init(fmt, w, h), Surface.init(fmt, w, h)
    bg = rng.integers(0, 256, a.data.size, dtype=np.uint8)
    if fmt in ("rgba", "argb", "rgb", "xrgb"):
        q = bg.reshape(-1, 4)
        al = {"rgba": 3, "rgb": 3, "argb": 0, "xrgb": 0}[fmt]
        q[:] = np.minimum(q, q[:, al:al + 1])
    a.data[:] = b.data[:] = bg
    ops = [Operation("dst_in", dst=src, src=mask), Operation(op)]
    assert gpu.composite(a, 0, 0, ops, precision) == abi.OK and oracle.composite(b, 0, 0, ops, precision) == abi.OK
    assert np.array_equal(a.numpy(), b.numpy()), (fmt, w, h, op, precision)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("fmt", ["rgba", "argb", "rgb", "xrgb", "alpha8", "alpha4", "alpha2", "alpha1"])
def test_pixel_source(gpu, oracle, fmt, size):
    src = Pattern.from_pixel(Pixel.rgba(90, 30, 140, 170))
    for op in ("src_over", "dst_out", "xor", "multiply", "clear"):
        for precision in ("integer", "float"):
            _check(gpu, oracle, fmt, *size, src, op, precision)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("kind", ["linear", "radial", "conic"])
@pytest.mark.parametrize("fmt", ["xrgb", "alpha8", "alpha4", "alpha1"])
def test_gradient_source(gpu, oracle, fmt, kind, size):
    w, h = size
    g = {"linear": lambda: Gradient.linear(0, 0, w, h, method="hsl"),
         "radial": lambda: Gradient.radial(w / 2, h / 2, 1, w / 2, h / 2, w, method="srgb"),
         "conic": lambda: Gradient.conic(w / 3, h / 2, 0.4, method="linear_rgb")}[kind]()
    g.add_stop(0.0, Color.rgb(1, 0, 0.3, 1)).add_stop(0.6, Color.rgb(0, 1, 0.5, 0.4)).add_stop(1.0, Color.rgb(0, 0, 1, 0.1))
    for src in (Pattern.from_gradient(g), Pattern.dither("blue_noise", g, 8)):
        for op in ("src_over", "multiply"):
            _check(gpu, oracle, fmt, w, h, src, op, "integer")


@pytest.mark.parametrize("size", SIZES)
def test_alpha8_layer(gpu, oracle, size):
    w, h = size
    rng = np.random.default_rng(w)
    for op in ("src_over", "xor", "dst_out", "multiply", "screen", "src", "plus"):
        for x, y in ((0, 0), (2, 1), (-1, 0)):
            a, b, s = Surface.init("alpha8", w + 5, h + 3), Surface.init("alpha8", w + 5, h + 3), Surface.init("alpha8", w, h)
            a.data[:] = b.data[:] = rng.integers(0, 256, a.data.size, dtype=np.uint8)
            s.data[:] = rng.integers(0, 256, s.data.size, dtype=np.uint8)
            src = [Operation(op, src=s)]
            assert gpu.composite(a, x, y, src) == abi.OK and oracle.composite(b, x, y, src) == abi.OK
            assert np.array_equal(a.numpy(), b.numpy()), (size, op, x, y)
