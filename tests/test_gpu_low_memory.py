"""Calls whose scratch in its usual, larger form does not fit the device any
more: they are drawn from the smaller form.  The device's memory is taken up
to a margin that holds the smaller form and not the larger one."""
import contextlib
import gc

import numpy as np
import pytest

from backends import StrokeOracle
from z2d_gb300 import abi, painter
from z2d_gb300.native import Context
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import NODE_DTYPE, FillOptions, Pattern, Pixel, StrokeOptions

pytestmark = pytest.mark.gpu
GB = 1 << 30


@contextlib.contextmanager
def only_free(n_bytes):
    """All but n_bytes of the device's free memory is taken."""
    torch = pytest.importorskip("torch")
    gc.collect()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - n_bytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def _stripes(x0, n, h):
    """n upright stripes of one pixel, every second column from x0, h rows."""
    p = Path()
    for k in range(n):
        x = x0 + 2 * k
        p.move_to(x, 0).line_to(x + 1, 0).line_to(x + 1, h).line_to(x, h).close()
    return p.to_array()


@pytest.mark.parametrize("fmt,op,many", [("alpha8", "src_over", False), ("rgba", "xor", False), ("alpha8", "src_over", True)])
def test_bins_of_indices(oracle, fmt, op, many):
    """400 fills of 128 stripes on a 256-column surface of 4,096 rows (and a
    second surface): 105 M entries are 3.4 GB of records, 0.4 of indices."""
    torch = pytest.importorskip("torch")
    w, h, n = 256, 4096, 400
    nodes, opts = [_stripes(x0, 128, h) for x0 in (0, 1)], FillOptions(operator=op)
    fills = [(Pattern.from_pixel(Pixel.rgba(k % 60, 40, 20, 90 + k % 100)), nodes[k % 2], opts) for k in range(n)]
    dev, ref = Surface.init(fmt, w, h).to_device("cuda"), Surface.init(fmt, w, 8)
    small = Surface.init(fmt, 40, 8).to_device("cuda")
    for pat, nd, o in fills:
        assert oracle.fill(ref, pat, nd, o) == abi.OK
    ctx = Context(0)
    with only_free(3 * GB):
        if many:
            painter.fill_jobs([(small, fills[:1]), (dev, fills)], ctx=ctx)
        else:
            painter.fill_batch(dev, fills, ctx=ctx)
        ctx.synchronize()
        ctx.close()
    got = dev.to_host().pixels()
    want = ref.pixels()
    assert np.array_equal(got, np.broadcast_to(want[:1], got.shape))
    if many:
        one = Surface.init(fmt, 40, 8)
        assert oracle.fill(one, *fills[0]) == abi.OK
        assert np.array_equal(small.to_host().numpy(), one.numpy())


def test_tiles_not_sorted():
    """16 surfaces of one column and 2^21 bands each: 2.1 GB of records fit, the
    0.8 GB that sorting the tiles takes do not beside them."""
    torch = pytest.importorskip("torch")
    h = (1 << 23) - 1
    nodes = Path().move_to(0, 0).line_to(1, 0).line_to(1, h).line_to(0, h).close().to_array()
    pat = Pattern.from_pixel(Pixel.rgba(0, 0, 0, 200))
    dev = [Surface.init("alpha8", 1, h).to_device("cuda") for _ in range(16)]
    torch.cuda.synchronize()

    def draw(ctx):
        painter.fill_jobs([(d, [(pat, nodes, FillOptions())]) for d in dev], ctx=ctx)
    ctx = Context(0)
    ctx.set_raster(0, 0, 0)
    before = torch.cuda.mem_get_info()[0]
    draw(ctx)
    ctx.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    ctx = Context(0)
    ctx.set_raster(0, 1, 0)
    with only_free(used + GB // 4):
        draw(ctx)
        ctx.synchronize()
        ctx.close()
    twice = 200 + 200 - 200 * 200 // 255
    for k, d in enumerate(dev):
        other = int((d.data != twice).sum())
        assert other == 0, f"surface {k}"


def _scratch_of(call):
    """What a call leaves allocated on the device."""
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    ctx = Context(0)
    before = torch.cuda.mem_get_info()[0]
    call(ctx)
    ctx.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    return used


def _wave():
    return Path().move_to(4, 30).curve_to(10, -20, 30, 70, 36, 8).line_to(20, 20).line_to(5, 5).to_array()


def _stroke_beside(oracle, big, less):
    """A stroke `big` off the surface and a small one on it, with `less` bytes
    fewer than the first call of its kind took."""
    pytest.importorskip("torch")
    pat = Pattern.from_pixel(Pixel.rgba(10, 200, 70, 255))
    opts = [StrokeOptions(line_width=2), StrokeOptions(line_width=5, line_join="round", line_cap="round")]
    ref = Surface.init("rgba", 40, 40)
    assert StrokeOracle(oracle).stroke(ref, pat, _wave(), opts[1]) == abi.OK
    dev = [Surface.init("rgba", 40, 40).to_device("cuda") for _ in range(2)]

    def draw(k):
        return lambda ctx: painter.draw_jobs([(dev[k], [("stroke", pat, big, opts[0]), ("stroke", pat, _wave(), opts[1])])],
                                             ctx=ctx)
    used = _scratch_of(draw(0))
    ctx = Context(0)
    with only_free(used - less):
        draw(1)(ctx)
        ctx.synchronize()
        ctx.close()
    for d in dev:
        assert np.array_equal(d.to_host().numpy(), ref.numpy())


def test_stroke_without_kept_joins(oracle):
    """Strokes of some 20 M points: their joins are 80 bytes each."""
    one = Path().move_to(0, -2e5).curve_to(1e6, -4e6, 2e6, -1e5, 3e6, -4e6)
    points = sum(len(c) for c in painter.stroke_contours(one.to_array(), StrokeOptions(line_width=2))[0]) // 5
    p = Path()
    n = (20 << 20) // points + 1
    for k in range(n):
        p.move_to(0, -2e5).curve_to(1e6, -4e6, 2e6, -1e5, 3e6, -4e6)
    _stroke_beside(oracle, p.to_array(), 40 * points * n)


def test_stroke_with_a_lane_a_node(oracle):
    """9 M stroked nodes: their counts are 128 bytes each with 8 lanes a node,
    16 with one."""
    n = 9_000_000
    k = np.arange(n)
    big = np.zeros(n, NODE_DTYPE)
    big["tag"] = np.where(k == 0, abi.MOVE_TO, abi.LINE_TO)
    big["p"][:, 0], big["p"][:, 1] = 10.0 * (k % 2), -100.0 - k % 1000
    _stroke_beside(oracle, big, 64 * n)
