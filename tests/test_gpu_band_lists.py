"""The band lists of batches whose jobs have very different numbers of fills:
around the number up to which a warp lists a band, beside many jobs of one
fill and jobs that draw nothing."""
import numpy as np
import pytest

from z2d_gb300 import abi, painter
from z2d_gb300.native import Context
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import FillOptions, Pattern, Pixel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[511], [512], [513], [1, 513], [513, 1], [1, 513, 1, 512, 1, 900, 0, 1], [600, 0, 600]])
def test_jobs_of_many_and_few(oracle, counts):
    rng = np.random.default_rng(sum(counts))
    counts = [c for big in counts for c in (big, 0, 1, 1, 1, 1)] if len(counts) > 1 else counts
    ctx = Context(0)
    jobs, refs = [], []
    for n in counts:
        w, h = int(rng.integers(5, 300)), int(rng.integers(5, 40))
        fills = []
        for k in range(max(n, 1)):
            x, y = rng.uniform(-3, [w, h]) if n else (-500, -500)
            nodes = Path().move_to(x, y).line_to(x + rng.uniform(1, 9), y).line_to(x, y + rng.uniform(1, 9)).close()
            fills.append((Pattern.from_pixel(Pixel.rgba(k % 100, 60, 10, 120)), nodes.to_array(), FillOptions()))
        ref = Surface.init("rgba", w, h)
        for f in fills:
            assert oracle.fill(ref, *f) == abi.OK
        refs.append(ref)
        jobs.append((Surface.init("rgba", w, h).to_device("cuda"), fills))
    painter.fill_jobs(jobs, ctx=ctx)
    ctx.synchronize()
    ctx.close()
    for k, ((dev, _), ref) in enumerate(zip(jobs, refs)):
        assert np.array_equal(dev.to_host().numpy(), ref.numpy()), f"job {k}"
