"""Gradient colours decided in f32 (grad_f32.cuh) against the oracle, byte for
byte: every kind, interpolation space and dither on random and adversarial
gradients, as whole-surface mask batches (k_mask_grad), as plain composites
and as fills; channels on and beside half-integers, offsets on stops, equal
and nearly equal stops, clear stops, no root, focal points outside, the branch
cut and the wrap on pixel centres, transformations.  And the gamma's error on
every float (tests/gamma_device_check.cu)."""
import math
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

from backends import GpuBackend
from z2d_gb300 import abi
from z2d_gb300.path import Path
from z2d_gb300.surface import Surface
from z2d_gb300.types import Color, FillOptions, Gradient, Operation, Pattern

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
W, H = 260, 52


@pytest.fixture(scope="module")
def gpu():
    return GpuBackend()


def test_gamma_error():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "gamma_device_check")
        subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "z2d_gb300", "csrc"),
                        os.path.join(HERE, "gamma_device_check.cu"), "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def _check(gpu, oracle, g, what):
    rng = np.random.default_rng(1)
    mask = Surface.init("alpha8", W, H)
    mask.data[:] = rng.integers(0, 256, mask.data.size, dtype=np.uint8)
    bg = rng.integers(0, 256, (W * H, 4), dtype=np.uint8)
    bg[:, :3] = np.minimum(bg[:, :3], bg[:, 3:])
    p = Path()
    for q in ((-3, -2), (W + 5, 4), (W - 9, H + 3), (7, H - 2)):
        (p.line_to if p.to_array().size else p.move_to)(*q)
    p.close()
    for dither in ("none", "bayer", "blue_noise"):
        src = Pattern.from_gradient(g) if dither == "none" else Pattern.dither(dither, g, 8)
        for fmt in ("rgba", "rgb"):
            for ops in ([Operation("dst_in", dst=src, src=mask), Operation("src_over")], [Operation("src", src=src)]):
                a, b = Surface.init(fmt, W, H), Surface.init(fmt, W, H)
                a.data[:] = b.data[:] = bg.reshape(-1)
                assert gpu.composite(a, 0, 0, ops) == abi.OK and oracle.composite(b, 0, 0, ops) == abi.OK
                assert np.array_equal(a.numpy(), b.numpy()), (what, dither, fmt, len(ops))
        for aa in ("default", "supersample_4x", "none"):
            a, b = Surface.init("rgba", W, H), Surface.init("rgba", W, H)
            a.data[:] = b.data[:] = bg.reshape(-1)
            opts = FillOptions(anti_aliasing=aa, fill_rule="even_odd")
            assert gpu.fill(a, src, p.to_array(), opts) == abi.OK and oracle.fill(b, src, p.to_array(), opts) == abi.OK
            assert np.array_equal(a.numpy(), b.numpy()), (what, dither, aa)


def _geometry(rng, kind, method):
    if kind == "linear":
        return Gradient.linear(*rng.uniform(-100, 400, 4), method=method)
    if kind == "radial":
        x, y, r = rng.uniform(0, W), rng.uniform(0, H), rng.uniform(5, 200)
        far = rng.uniform(0, 1.6)  # beyond 1: the focal circle leaves the outer one
        return Gradient.radial(x, y, rng.uniform(0, 30), x + far * r * 0.7, y + far * r * 0.7, r, method=method)
    return Gradient.conic(rng.uniform(0, W), rng.uniform(0, H), rng.uniform(-7, 7), method=method)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("kind", ["linear", "radial", "conic"])
@pytest.mark.parametrize("method", ["linear_rgb", "srgb", "hsl"])
def test_random(gpu, oracle, seed, kind, method):
    rng = np.random.default_rng(100 * seed + len(kind) + 7 * len(method))
    g = _geometry(rng, kind, method)
    n = int(rng.integers(1, 7))
    offs = np.sort(rng.uniform(0, 1, n))
    if seed == 1:
        offs[-1] = offs[0]                       # equal stops
    if seed == 2:
        offs = offs[0] + np.arange(n) * 2e-7     # nearly equal ones
    for o in offs:
        a = 0.0 if seed == 3 and rng.random() < 0.4 else float(rng.uniform(0.01, 1))
        g.add_stop(float(o), Color.rgb(*map(float, rng.random(3)), a))
    if seed >= 4:
        t, s = rng.uniform(-3, 3), rng.uniform(0.2, 4)
        g.set_transformation((s * math.cos(t), s * math.sin(t), -math.sin(t), math.cos(t), *rng.uniform(-300, 300, 2)))
    _check(gpu, oracle, g, (seed, kind, method))


ADVERSARIAL = {
    "ties": lambda m: Gradient.linear(0, 0, 255, 0, method=m),          # 255 t = x + 1/2 on every pixel
    "half_steps": lambda m: Gradient.linear(0, 0, 510, 0, method=m),
    "stops_on_pixels": lambda m: Gradient.linear(0.5, 0, 128.5, 0, method=m),
    "tiny": lambda m: Gradient.linear(100, 20, 100.001, 20, method=m),
    "huge": lambda m: Gradient.linear(-1e7, -1e7, 1e7, 1e7, method=m),
    "void": lambda m: Gradient.linear(5, 5, 5, 5, method=m),
    "centre_on_pixel": lambda m: Gradient.radial(100.5, 20.5, 0, 100.5, 20.5, 60, method=m),
    "equal_circles": lambda m: Gradient.radial(60, 20, 30, 160, 20, 30, method=m),
    "a_zero": lambda m: Gradient.radial(60, 20, 10, 60, 70, 60, method=m),
    "no_root": lambda m: Gradient.radial(60, 20, 5, 200, 20, 20, method=m),
    "cut_on_row": lambda m: Gradient.conic(130.5, 25.5, 0.0, method=m),
    "wrap_on_row": lambda m: Gradient.conic(130.5, 25.5, math.pi, method=m),
    "far_conic": lambda m: Gradient.conic(-1e6, 1e6, 1.0, method=m),
}


@pytest.mark.parametrize("name", sorted(ADVERSARIAL))
@pytest.mark.parametrize("method", ["linear_rgb", "srgb"])
def test_adversarial(gpu, oracle, name, method):
    g = ADVERSARIAL[name](method)
    g.add_stop(0.0, Color.rgb(0, 0, 1, 1)).add_stop(0.25, Color.rgb(1, 0.5, 0, 1)).add_stop(0.5, Color.rgb(0, 1, 0.2, 1))
    g.add_stop(0.5, Color.rgb(1, 1, 1, 0.5)).add_stop(1.0, Color.rgb(0, 0, 0, 1))
    _check(gpu, oracle, g, name)
    g = ADVERSARIAL[name](method)
    g.add_stop(0.0, Color.rgb(0, 0, 0, 1)).add_stop(1.0, Color.rgb(1, 1, 1, 1))
    _check(gpu, oracle, g, name)


@pytest.mark.parametrize("size", [(1, 1), (31, 1), (33, 3), (37, 5), (255, 7), (1021, 3)])
def test_mask_sizes(gpu, oracle, size):
    """Whole-surface batches whose pixel count is no multiple of anything."""
    w, h = size
    rng = np.random.default_rng(w)
    g = Gradient.radial(w / 2, h / 2, 1, w / 2, h / 2, w, method="srgb")
    g.add_stop(0.0, Color.rgb(1, 0, 0.3, 1)).add_stop(1.0, Color.rgb(0, 1, 0.5, 0.4))
    mask = Surface.init("alpha8", w, h)
    mask.data[:] = rng.integers(0, 256, mask.data.size, dtype=np.uint8)
    for op in ("src_over", "xor", "multiply"):
        ops = [Operation("dst_in", dst=Pattern.dither("blue_noise", g, 8), src=mask), Operation(op)]
        a, b = Surface.init("argb", w, h), Surface.init("argb", w, h)
        assert gpu.composite(a, 0, 0, ops) == abi.OK and oracle.composite(b, 0, 0, ops) == abi.OK
        assert np.array_equal(a.numpy(), b.numpy()), (size, op)
