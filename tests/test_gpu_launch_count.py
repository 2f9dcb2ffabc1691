"""z2dgpu_ctx_launch_count against the kernels that the device ran, as the
profiler lists them: every launch is counted, and a call of one short fill is
one launch."""
import pytest

from z2d_gb300 import painter
from z2d_gb300.native import Context
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import Color, FillOptions, Gradient, Pattern, Pixel

pytestmark = pytest.mark.gpu


def _kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return [e.name for e in prof.events()
            if e.device_type == torch.autograd.DeviceType.CUDA and "Memcpy" not in e.name and "Memset" not in e.name]


@pytest.mark.parametrize("source", ["pixel", "gradient"])
@pytest.mark.parametrize("segments", [8, 1200])
def test_small_calls_are_one_launch(source, segments):
    torch = pytest.importorskip("torch")
    pat = Pattern.from_pixel(Pixel.rgba(90, 10, 10, 255))
    if source == "gradient":
        g = Gradient.linear(0, 0, 300, 300)
        g.add_stop(0.0, Color.rgb(1, 0, 0, 1)).add_stop(1.0, Color.rgb(0, 1, 0, 0.5))
        pat = Pattern.from_gradient(g)
    p = Path().move_to(150, 10)
    for k in range(segments):
        p.line_to(10 + (k * 37) % 280, 20 + (k * 53) % 270)
    nodes, s, ctx = p.close().to_array(), Surface.init("rgba", 300, 300).to_device("cuda"), Context(0)
    torch.cuda.synchronize()
    painter.fill(s, pat, nodes, FillOptions(), ctx=ctx)
    # (the profiler's first run may list nothing)
    if not any([_kernels(lambda: painter.fill(s, pat, nodes, FillOptions(), ctx=ctx)) for _ in range(2)]):
        pytest.skip("the profiler lists no kernels here")
    n0 = ctx.launch_count
    names = _kernels(lambda: painter.fill(s, pat, nodes, FillOptions(), ctx=ctx))
    assert len(names) == ctx.launch_count - n0 == 1, names
    ctx.close()
