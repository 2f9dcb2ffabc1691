"""k_fill_scan's runs of segments against the oracle, byte for byte: paths
whose moves, closes and starts after a close fall on every position of the
warp's 32 nodes, repeated points, open chains, and band lists of few and of
many fills a job."""
import numpy as np
import pytest

from z2d_gb300 import abi, painter
from z2d_gb300.native import default_context
from z2d_gb300.surface import Surface
from z2d_gb300.types import NODE_DTYPE, FillOptions, Pattern, Pixel

pytestmark = pytest.mark.gpu
W, H = 90, 50
PIX = Pattern.from_pixel(Pixel.rgba(60, 20, 90, 170))


def _path(rng, lengths, bare):
    """Subpaths of the given segment counts; with `bare`, every other one
    starts at the close_path before it instead of a move_to."""
    out = []

    def node(tag, *p):
        a = np.zeros((), NODE_DTYPE)
        a["tag"] = tag
        a["p"][:len(p)] = p
        out.append(a)

    def pt():
        return float(rng.uniform(-5, W + 5)), float(rng.uniform(-5, H + 5))

    start = pt()
    for i, n in enumerate(lengths):
        if i == 0 or not (bare and i % 2):
            start = pt()
            node(abi.MOVE_TO, *start)
        last = start
        for _ in range(n):
            p = last if rng.random() < 0.15 else pt()  # repeated points among them
            if rng.random() < 0.3:
                node(abi.CURVE_TO, *pt(), *pt(), *p)
            else:
                node(abi.LINE_TO, *p)
            last = p
        node(abi.CLOSE_PATH)
    node(abi.MOVE_TO, *start)
    return np.array(out, NODE_DTYPE)


def _draw(oracle, fills):
    a, b = Surface.init("rgba", W, H), Surface.init("rgba", W, H)
    off = _path(np.random.default_rng(0), [4200], False)  # sends the call to the pipeline, off the surface
    off["p"] -= 5000
    painter.fill_batch(a, fills + [(PIX, off, FillOptions())])
    for f in fills:
        assert oracle.fill(b, *f) == abi.OK
    assert np.array_equal(a.numpy(), b.numpy())


@pytest.mark.parametrize("n", [1, 2, 3, 27, 28, 29, 30, 31, 32, 33, 60, 61, 62, 63, 64, 65, 100])
@pytest.mark.parametrize("bare", [False, True])
def test_positions(oracle, n, bare):
    rng = np.random.default_rng(n)
    _draw(oracle, [(PIX, _path(rng, lengths, bare), FillOptions(fill_rule=rule))
                   for lengths in ([n], [n, 1, n], [3, n, 2, n, 5], [1, 1, n, 1, 1]) for rule in ("non_zero", "even_odd")])


@pytest.mark.parametrize("n", [31, 33, 255, 257, 700])
def test_many_fills(oracle, n):
    rng = np.random.default_rng(n)
    _draw(oracle, [(PIX, _path(rng, [3], False), FillOptions(fill_rule="even_odd")) for _ in range(n)])


def test_jobs_of_few_fills(oracle):
    rng = np.random.default_rng(9)
    ctx = default_context()
    jobs, refs = [], []
    for k in range(40):
        fills = [(PIX, _path(rng, [int(rng.integers(1, 70))], False), FillOptions()) for _ in range(k % 4)]
        ref = Surface.init("rgba", W, H)
        for f in fills:
            assert oracle.fill(ref, *f) == abi.OK
        refs.append(ref)
        jobs.append((Surface.init("rgba", W, H).to_device(), fills))
    painter.fill_jobs(jobs, ctx=ctx)
    ctx.synchronize()
    for (s, _), ref in zip(jobs, refs):
        assert np.array_equal(s.numpy(), ref.numpy())
