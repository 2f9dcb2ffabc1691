"""One surface composited onto another at an offset (k_layer) against the
oracle, byte for byte: every integer operator, the 4-byte formats crossed,
offsets negative and beyond the right and bottom edge, widths around the
warp's 32 and 128 pixels, single rows and columns, a surface onto itself, and
the shapes that keep the general kernels (alpha formats, float operators)."""
import numpy as np
import pytest

from backends import GpuBackend
from z2d_gb300 import abi
from z2d_gb300.surface import Surface
from z2d_gb300.types import Operation

pytestmark = pytest.mark.gpu
INT_OPS = [o for o in abi.OPERATORS if o not in abi.FLOAT_ONLY_OPS]


@pytest.fixture(scope="module")
def gpu():
    return GpuBackend()


def _surface(fmt, w, h, seed):
    s = Surface.init(fmt, w, h)
    d = np.random.default_rng(seed).integers(0, 256, s.data.size, dtype=np.uint8)
    if fmt in ("rgba", "argb"):
        d = d.reshape(-1, 4)
        d[:, :3] = np.minimum(d[:, :3], d[:, 3:])
    s.data[:] = d.reshape(-1)
    return s


def _check(gpu, oracle, df, sf, dsize, ssize, x, y, op, what):
    a, b, s = _surface(df, *dsize, 1), _surface(df, *dsize, 1), _surface(sf, *ssize, 2)
    assert gpu.composite(a, x, y, [Operation(op, src=s)]) == abi.OK
    assert oracle.composite(b, x, y, [Operation(op, src=s)]) == abi.OK
    assert np.array_equal(a.numpy(), b.numpy()), what


@pytest.mark.parametrize("op", INT_OPS)
def test_operators(gpu, oracle, op):
    for df in ("rgba", "xrgb"):
        for sf in ("rgba", "argb", "rgb"):
            _check(gpu, oracle, df, sf, (150, 9), (133, 7), 5, 1, op, (op, df, sf))


@pytest.mark.parametrize("df", ["rgba", "argb", "rgb", "xrgb", "alpha8", "alpha4"])
@pytest.mark.parametrize("sf", ["rgba", "argb", "rgb", "xrgb", "alpha8"])
def test_formats(gpu, oracle, df, sf):
    for op in ("src_over", "xor", "hue"):
        _check(gpu, oracle, df, sf, (70, 6), (64, 9), 3, -2, op, (op, df, sf))


@pytest.mark.parametrize("w", [1, 31, 32, 33, 127, 128, 129, 257])
def test_widths_and_offsets(gpu, oracle, w):
    for x, y in ((0, 0), (1, 0), (-1, 2), (7, -3), (200, 3), (259, 4), (-w + 1, 4), (-w, 0), (260, 0), (0, 5)):
        _check(gpu, oracle, "rgba", "rgba", (260, 5), (w, 4), x, y, "src_over", (w, x, y))


def test_onto_itself(gpu, oracle):
    a, b = _surface("rgba", 130, 7, 3).to_device(), _surface("rgba", 130, 7, 3)
    assert gpu.composite(a, 0, 0, [Operation("src_over", src=a)]) == abi.OK
    gpu.ctx.synchronize()
    assert oracle.composite(b, 0, 0, [Operation("src_over", src=_surface("rgba", 130, 7, 3))]) == abi.OK
    assert np.array_equal(a.numpy(), b.numpy())
