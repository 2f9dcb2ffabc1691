"""Calls whose scratch in its usual, larger form does not fit the device any
more: they are drawn from the smaller form.  The device's memory is taken up
to a margin that holds the smaller form and not the larger one."""
import contextlib
import gc

import numpy as np
import pytest

from z2d_gb300 import abi, painter
from z2d_gb300.native import Context
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import FillOptions, Pattern, Pixel

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
