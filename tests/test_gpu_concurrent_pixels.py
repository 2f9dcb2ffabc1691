"""A fill writes the pixels it covers and no others: two contexts, each on its
own stream, draw different pixels of one device surface at the same time.

The first draws a long batch on pixel column 0 (every row of it is at work
for milliseconds), the second meanwhile columns 1 to 31 of the same 32
pixels; both drawings must be there afterwards.
"""
import numpy as np
import pytest

from z2d_gb300 import abi, painter
from z2d_gb300.native import Context
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import Color, FillOptions, Gradient, Pattern, Pixel

pytestmark = pytest.mark.gpu

W, H, N = 32, 16, 6000


def _rect(x0, x1):
    return Path().move_to(x0, 0).line_to(x1, 0).line_to(x1, H).line_to(x0, H).close().to_array()


def _gradient():
    g = Gradient.linear(0, 0, 0, H)
    g.add_stop(0.0, Color.rgb(1, 0, 0, 0.5)).add_stop(1.0, Color.rgb(0, 0, 1, 1))
    return Pattern.from_gradient(g)


@pytest.mark.parametrize("fmt,source,opts", [
    ("rgba", "pixel", {}),
    ("rgba", "pixel", {"anti_aliasing": "none"}),
    ("rgba", "pixel", {"anti_aliasing": "supersample_4x"}),
    ("rgba", "gradient", {}),
    ("rgba", "pixel", {"operator": "multiply"}),
    ("xrgb", "pixel", {}),
    ("alpha8", "pixel", {}),
    ("alpha4", "pixel", {}),
    ("alpha1", "pixel", {"operator": "xor"}),
])
def test_two_streams_one_block(oracle, fmt, source, opts):
    torch = pytest.importorskip("torch")
    opts = FillOptions(**opts)
    pat = _gradient() if source == "gradient" else Pattern.from_pixel(Pixel.rgba(60, 90, 120, 130))
    other = Pattern.from_pixel(Pixel.rgba(200, 10, 30, 255))
    slow = [(pat, _rect(0, 1), opts)] * N
    dev, ref = Surface.init(fmt, W, H).to_device("cuda"), Surface.init(fmt, W, H)
    torch.cuda.synchronize()
    a, b = Context(0), Context(0)
    painter.fill_batch(dev, slow, ctx=a)
    painter.fill(dev, other, _rect(1, W), FillOptions(), ctx=b)
    b.synchronize()
    a.synchronize()
    for p, nodes, o in slow + [(other, _rect(1, W), FillOptions())]:
        assert oracle.fill(ref, p, nodes, o) == abi.OK
    got, want = dev.to_host().numpy(), ref.numpy()
    a.close()
    b.close()
    assert np.array_equal(got, want), f"{int((got != want).sum())} values differ"
