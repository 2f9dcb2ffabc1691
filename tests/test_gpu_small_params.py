"""Calls whose tables travel as kernel parameters and, above that size, by a
copy: closed polygons around the change (their tables grow by some 100 bytes
a corner), with pixel and gradient sources, on one surface and, in turn, on
two, without a synchronisation between the calls, against the oracle."""
import math

import numpy as np
import pytest
import torch

from backends import GpuBackend
from z2d_gb300 import abi, painter
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import Color, FillOptions, Gradient, Pattern, Pixel

pytestmark = pytest.mark.gpu


def _polygon(n, cx, cy, r, turns):
    p = Path()
    for k in range(n):
        t = 2 * math.pi * turns * k / n
        q = (cx + r * (1 + 0.3 * (k % 3)) / 1.6 * math.cos(t), cy + r * math.sin(t))
        (p.line_to if k else p.move_to)(*q)
    p.close()
    return p.to_array()


@pytest.mark.parametrize("n", [3, 8, 16, 24, 32, 40, 48, 56, 64, 72, 80, 96, 128, 400])
@pytest.mark.parametrize("size", [(20, 7), (301, 211)])
def test_sizes(oracle, n, size):
    w, h = size
    gpu = GpuBackend()
    g = Gradient.linear(0, 0, w, h).add_stop(0, Color.rgb(1, 0, 0, 1)).add_stop(1, Color.rgb(0, 0.4, 1, 0.5))
    dev = [Surface.init("rgba", w, h).to_device() for _ in range(2)]
    want = [Surface.init("rgba", w, h) for _ in range(2)]
    for k in range(6):
        pat = Pattern.from_gradient(g) if k == 3 else Pattern.from_pixel(Pixel.rgba(30 * k, 100, 50, 200))
        nodes = _polygon(n + k, w * 0.5, h * 0.4 + k, 0.45 * min(w, h) + 2 * k, 1 + k % 3)
        opts = FillOptions(fill_rule="even_odd" if k % 2 else "non_zero")
        painter.fill(dev[k % 2], pat, nodes, opts, ctx=gpu.ctx)
        assert oracle.fill(want[k % 2], pat, nodes, opts) == abi.OK
    torch.cuda.synchronize()
    for a, b in zip(dev, want):
        assert np.array_equal(a.numpy(), b.numpy()), (n, size)
