"""The schedule tuner keeps the rasteriser's modes apart: a gradient batch does
not take the choice measured on a pixel batch of the same size, and a saved
table of choices without a mode is not taken."""
import json
import os
import subprocess
import sys

import pytest

from z2d_gb300 import painter
from z2d_gb300.native import Context
from z2d_gb300.surface import Surface
from z2d_gb300.types import Color, FillOptions, Gradient, Pattern, Pixel
from z2d_gb300.workloads import random_fills

pytestmark = pytest.mark.gpu

W, H = 900, 333
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _fills(source):
    pat = Pattern.from_pixel(Pixel.rgba(40, 30, 20, 100))
    if source == "gradient":
        g = Gradient.linear(0, 0, W, H)
        g.add_stop(0.0, Color.rgb(1, 0, 0, 0.5)).add_stop(1.0, Color.rgb(0, 0, 1, 1))
        pat = Pattern.from_gradient(g)
    return [(pat, nodes, FillOptions()) for _, nodes, _ in random_fills(seed=5, n=90, w=W, h=H, side_lo=200, side_hi=300)]


def _draw(ctx, source, passes):
    s = Surface.init("rgba", W, H)
    for _ in range(passes):
        painter.fill_batch(s, _fills(source), ctx=ctx)
    return ctx.raster_tuning()["decided"]


def test_modes_are_tuned_apart():
    ctx = Context(0)
    decided = _draw(ctx, "pixel", 9)
    if decided == -1:
        pytest.skip("autotuning is off (Z2D_TUNE=off)")
    assert decided == 1
    assert _draw(ctx, "gradient", 1) == 0
    assert _draw(ctx, "gradient", 9) == 1
    assert _draw(ctx, "pixel", 1) == 1
    ctx.close()


@pytest.mark.parametrize("mode", [None, 1])
def test_saved_choices(tmp_path, mode):
    """A saved choice for every key, with the pixel batch's mode or none."""
    path = tmp_path / "raster_tune.json"
    lines = []
    for tiles in range(20):
        for load in range(20):
            d = {"multi": 0, "mode": mode, "tiles": tiles, "load": load, "ctas": 0, "order": 0, "cta_items": 1, "ms": 0.5}
            lines.append(json.dumps({k: v for k, v in d.items() if v is not None}))
    path.write_text("\n".join(lines) + "\n")
    code = ("import sys; sys.path[:0] = [%r, %r]; import test_gpu_tune_modes as t; from z2d_gb300.native import Context; "
            "c = Context(0); print('decided', t._draw(c, 'pixel', 1)); c.close()" % (ROOT, os.path.join(ROOT, "tests")))
    env = dict(os.environ, Z2D_TUNE_FILE=str(path))
    env.pop("Z2D_TUNE", None)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stdout + r.stderr
    assert f"decided {0 if mode is None else 1}" in r.stdout
