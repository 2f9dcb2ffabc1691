"""What a program that draws with this framework has it do: single fills and
strokes, batches of fills on one surface, batches over many surfaces,
compositing of whole layers and the export of PNG image data, each through the package's public
entry points.

Every output is a surface's bytes (or the exported rows'), drawn in integer or
IEEE arithmetic that z2d prescribes bit for bit.
"""
import ctypes as C
import math

import numpy as np
import torch

from z2d_gb300 import abi, compositor, painter, png
from z2d_gb300.batch import PackedBatch, PackedDrawBatch
from z2d_gb300.surface import Surface
from z2d_gb300.types import NODE_DTYPE, Color, FillOptions, Gradient, Operation, Pattern, Pixel, StrokeOptions
from z2d_gb300.workloads import random_path_batch, star_300

# The share of a random path's bounding box that its fill covers, about.
COVERED = 0.4
BLEND_FLOPS = 8  # a multiply and an add for each of four channels


def listed():
    return [
        # The smallest call: an icon-sized surface and one closed polygon.
        {"name": "star_300", "kind": "star", "format": "rgba"},
        # One painter.fill as a program issues them one by one: a path of 40 lines and curves on a large canvas.
        {"name": "fill_path", "kind": "fill", "w": 4096, "h": 4096, "format": "rgba", "segments": 40, "side": 600.0,
         "source": "pixel", "aa": "default"},
        # A drawing of 2,000 random paths submitted at once: the benchmark's workload.
        {"name": "batch_2000", "kind": "batch", "w": 4096, "h": 4096, "format": "rgba", "n": 2000, "side_lo": 16.0,
         "side_hi": 1024.0, "seg_hi": 64, "source": "pixel", "aa": "default", "op": "src_over"},
        # An illustration with gradient paints on an odd-sized window surface.
        {"name": "batch_gradients", "kind": "batch", "w": 1999, "h": 1333, "format": "argb", "n": 240, "side_lo": 16.0,
         "side_hi": 512.0, "seg_hi": 24, "source": "gradient", "aa": "default", "op": "src_over"},
        # A coverage mask drawn with supersampling on an alpha surface.
        {"name": "batch_mask_ssaa", "kind": "batch", "w": 1025, "h": 1023, "format": "alpha8", "n": 300, "side_lo": 8.0,
         "side_hi": 400.0, "seg_hi": 32, "source": "pixel", "aa": "supersample_4x", "op": "src_over"},
        # One painter.stroke: a wide polyline of lines and curves with round joins and caps.
        {"name": "stroke_path", "kind": "stroke", "w": 2048, "h": 2048, "format": "rgba", "segments": 48, "side": 1500.0,
         "width": 7.5, "join": "round", "cap": "round", "dashed": False},
        # A tile renderer's pass: many surfaces of unlike sizes, fills and (solid and dashed) strokes mixed.
        {"name": "jobs_mixed", "kind": "jobs", "n": 320, "side_lo": 16, "side_hi": 2048, "paths_hi": 200, "strokes": 0.3},
        # A text renderer's pass: glyph outlines, each on a small surface of its own.
        {"name": "glyphs_1024", "kind": "glyphs", "n": 1024, "box": 64, "cubics_lo": 20, "cubics_hi": 200},
        # Painting a full canvas through a mask, the largest surface in use.
        {"name": "mask_8192", "kind": "mask", "w": 8192, "h": 8192, "format": "rgba", "source": "pixel",
         "method": "linear_rgb", "dither": "none", "op": "src_over", "precision": "integer"},
        # A radial sRGB gradient with dithering painted through a mask.
        {"name": "mask_radial_srgb", "kind": "mask", "w": 3840, "h": 2160, "format": "rgba", "source": "radial",
         "method": "srgb", "dither": "blue_noise", "op": "src_over", "precision": "integer"},
        # Composing one layer onto another at an offset, as a scene's layers are flattened.
        {"name": "layer_over", "kind": "layer", "w": 3840, "h": 2160, "sw": 2563, "sh": 1441, "x": 333, "y": 217,
         "format": "rgba", "op": "src_over"},
        # The image data of a finished drawing, as a PNG encoder takes it.
        {"name": "png_rows", "kind": "png", "w": 2561, "h": 1441, "format": "rgba", "profile": "srgb"},
    ]


FORMATS = ["rgba", "rgba", "argb", "rgb", "xrgb", "alpha8", "alpha4", "alpha1"]
OPERATORS = ["src_over", "src_over", "src_over", "dst_over", "dst_out", "xor", "plus", "multiply", "screen"]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["fill", "batch", "batch", "stroke", "jobs", "glyphs", "mask", "mask", "layer", "png"])
    if kind == "fill":
        w, h = int(_log(rng, 64, 4096)), int(_log(rng, 64, 4096))
        return {"kind": kind, "w": w, "h": h, "format": rng.choice(FORMATS[:6]), "segments": rng.randint(3, 64),
                "side": round(_log(rng, 16, max(17.0, min(w, h) * 0.5)), 1),
                "source": rng.choice(["pixel", "pixel", "gradient"]),
                "aa": rng.choice(["default", "default", "supersample_4x", "none"])}
    if kind == "batch":
        w, h = int(_log(rng, 200, 4096)), int(_log(rng, 200, 4096))
        s = min(w, h)
        return {"kind": kind, "w": w, "h": h, "format": rng.choice(FORMATS), "n": int(_log(rng, 16, 1500)),
                "side_lo": 8.0, "side_hi": round(rng.uniform(s / 16, s / 4), 1), "seg_hi": rng.randint(8, 64),
                "source": rng.choice(["pixel", "pixel", "gradient"]),
                "aa": rng.choice(["default", "default", "default", "supersample_4x", "none"]),
                "op": rng.choice(OPERATORS)}
    if kind == "stroke":
        w, h = int(_log(rng, 100, 4096)), int(_log(rng, 100, 4096))
        return {"kind": kind, "w": w, "h": h, "format": rng.choice(FORMATS[:6]), "segments": rng.randint(2, 64),
                "side": round(_log(rng, 32, max(33.0, min(w, h) * 0.9)), 1), "width": round(rng.uniform(0.5, 20.0), 2),
                "join": rng.choice(["miter", "round", "bevel"]), "cap": rng.choice(["butt", "round", "square"]),
                "dashed": rng.random() < 0.3}
    if kind == "jobs":
        return {"kind": kind, "n": int(_log(rng, 8, 256)), "side_lo": 16, "side_hi": int(_log(rng, 64, 2048)),
                "paths_hi": rng.randint(5, 200), "strokes": round(rng.choice([0.0, 0.3, rng.uniform(0.0, 0.5)]), 3)}
    if kind == "glyphs":
        return {"kind": kind, "n": int(_log(rng, 4, 2048)), "box": rng.randint(16, 96), "cubics_lo": 20,
                "cubics_hi": rng.randint(30, 200)}
    if kind == "mask":
        fmt = rng.choice(FORMATS)
        source = rng.choice(["pixel", "pixel", "linear", "radial", "conic"])
        return {"kind": kind, "w": int(_log(rng, 64, 8192)), "h": int(_log(rng, 64, 8192)), "format": fmt,
                "source": source, "method": rng.choice(["linear_rgb", "srgb", "hsl"]),
                "dither": "none" if source == "pixel" else rng.choice(["none", "none", "bayer", "blue_noise"]),
                "op": rng.choice(OPERATORS),
                "precision": "float" if fmt == "rgba" and rng.random() < 0.25 else "integer"}
    if kind == "layer":
        w, h = int(_log(rng, 64, 4096)), int(_log(rng, 64, 4096))
        sw, sh = max(16, int(w * rng.uniform(0.2, 1.0))), max(16, int(h * rng.uniform(0.2, 1.0)))
        return {"kind": kind, "w": w, "h": h, "sw": sw, "sh": sh, "x": rng.randint(0, w - sw), "y": rng.randint(0, h - sh),
                "format": rng.choice(FORMATS[:5]), "op": rng.choice(OPERATORS)}
    return {"kind": "png", "w": int(_log(rng, 64, 4096)), "h": int(_log(rng, 64, 4096)), "format": rng.choice(FORMATS),
            "profile": rng.choice(["none", "srgb", "linear"])}


def work(case):
    kind, bpp = case["kind"], abi.FORMAT_BITS[abi.FORMAT_NAMES.index(case.get("format", "rgba"))] / 8
    if kind == "star":
        return {"bytes": 2 * bpp * 232 * 254, "flops": BLEND_FLOPS * 0.28 * 300 * 300}
    if kind in ("fill", "stroke"):
        box = min(case["side"], case["w"]) * min(case["side"], case["h"])
        part = COVERED if kind == "fill" else min(COVERED, 0.4 * case["segments"] * case["width"] / case["side"])
        return {"bytes": 56.0 * (case["segments"] + 3) + 2 * bpp * part * box, "flops": BLEND_FLOPS * part * box}
    if kind == "batch":
        lo, hi = case["side_lo"], case["side_hi"]
        boxes = case["n"] * (hi * hi + hi * lo + lo * lo) / 3
        nodes = case["n"] * ((3 + case["seg_hi"]) / 2 + 3)
        return {"bytes": 56.0 * nodes + 2 * bpp * min(case["w"] * case["h"], COVERED * boxes),
                "flops": BLEND_FLOPS * COVERED * boxes}
    if kind == "jobs":
        sizes = _job_sizes(case)
        px = float((sizes[:, 0] * sizes[:, 1]).sum())
        n = case["n"] * (1 + case["paths_hi"]) / 2
        return {"bytes": 8 * px + 56 * 37.0 * n,
                "flops": BLEND_FLOPS * COVERED * 0.085 * px * (1 + case["paths_hi"]) / 2}
    if kind == "glyphs":
        px = case["n"] * case["box"] ** 2
        return {"bytes": 8.0 * px * COVERED + 56.0 * case["n"] * ((case["cubics_lo"] + case["cubics_hi"]) / 2 + 3),
                "flops": BLEND_FLOPS * COVERED * px}
    if kind == "mask":
        px = case["w"] * case["h"]
        return {"bytes": (2 * bpp + 1) * px, "flops": (BLEND_FLOPS + 4 + (20 if case["source"] != "pixel" else 0)) * px}
    if kind == "layer":
        px = case["sw"] * case["sh"]
        return {"bytes": 3 * bpp * px, "flops": BLEND_FLOPS * px}
    return {"bytes": 2 * bpp * case["w"] * case["h"], "flops": 4.0 * case["w"] * case["h"]}


def exact(case, seed):
    return None  # every output is bytes


# ------------------------------------------------------------------ inputs
def _pixels(seed, n):
    """n random premultiplied RGBA pixels in device memory."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    a = torch.randint(0, 256, (n,), device="cuda", generator=g, dtype=torch.int32)
    rgb = torch.randint(0, 256, (n, 3), device="cuda", generator=g, dtype=torch.int32) * (a[:, None] + 1) // 256
    return torch.cat([rgb, a[:, None]], 1).to(torch.uint8).reshape(-1)


def _surface(seed, fmt, w, h):
    """A device surface that has been drawn on: premultiplied pixels, or random alpha values."""
    f = abi.FORMAT_NAMES.index(fmt)
    if f == abi.FORMAT_RGBA or f == abi.FORMAT_ARGB:
        return Surface(fmt, w, h, _pixels(seed, w * h))  # (ARGB stores the alpha byte last too)
    n = abi.surface_bytes(f, w, h)
    n = (n + 3) // 4 * 4 if f >= abi.FORMAT_ALPHA4 else n
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    data = torch.randint(0, 256, (n,), device="cuda", generator=g, dtype=torch.uint8)
    if f in (abi.FORMAT_RGB, abi.FORMAT_XRGB):
        data.view(-1, 4)[:, 3] = 0
    return Surface(fmt, w, h, data)


def _colours(rng, n):
    a = rng.integers(32, 256, n)
    rgb = (rng.random((n, 3)) * (a[:, None] + 1)).astype(np.int64)
    return np.concatenate([np.minimum(rgb, a[:, None]), a[:, None]], 1).astype(np.uint8)


def _color(rng, alpha_lo=0.3):
    r, g, b = (float(v) for v in rng.random(3))
    return Color.rgb(r, g, b, float(rng.uniform(alpha_lo, 1.0)))


def _gradient(rng, kind, method, x0, y0, x1, y1, stops):
    """A gradient that runs over the box (x0, y0)-(x1, y1)."""
    cx, cy, r = (x0 + x1) / 2, (y0 + y1) / 2, max(x1 - x0, y1 - y0) / 2
    if kind == "linear":
        g = Gradient.linear(x0, y0, x1, y1, method=method)
    elif kind == "radial":
        g = Gradient.radial(cx - r / 8, cy, r / 50, cx, cy + r / 9, r, method=method)
    else:
        g = Gradient.conic(cx, cy, float(rng.uniform(0, 6)), method=method)
    for k in range(stops):
        g.add_stop(k / (stops - 1), _color(rng))
    return g


def _source(rng, kind, nodes):
    if kind == "pixel":
        return Pattern.from_pixel(Pixel.rgba(*map(int, _colours(rng, 1)[0])))
    p = nodes["p"][nodes["tag"] != abi.CLOSE_PATH][:, :2]
    (x0, y0), (x1, y1) = p.min(0), p.max(0)
    which = ("linear", "radial", "conic")[int(rng.integers(0, 3))]
    method = ("linear_rgb", "srgb", "hsl")[int(rng.integers(0, 3))]
    return Pattern.from_gradient(_gradient(rng, which, method, float(x0), float(y0), float(x1) + 1, float(y1) + 1,
                                           int(rng.integers(2, 6))))


def _one_path(rng, case):
    nodes, _, _ = random_path_batch(rng, 1, case["w"], case["h"], case["side"], case["side"], case["segments"],
                                    case["segments"])
    return nodes


def _dashes(rng):
    return tuple(rng.uniform(1.0, 40.0, int(rng.integers(2, 7))))


def _job_sizes(case):
    """The job surfaces' sides: log-uniform, the same for every seed."""
    rng = np.random.default_rng([case["n"], case["side_lo"], case["side_hi"]])
    return np.round(np.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"]), (case["n"], 2)))).astype(int)


def _atlas(seed, sizes):
    """Job surfaces as parts of one device buffer of drawn pixels."""
    starts, total = [], 0
    for w, h in sizes:
        starts.append(total)
        total += (int(w) * int(h) * 4 + 255) // 256 * 256
    data = _pixels(seed, total // 4)
    return data, [Surface("rgba", int(w), int(h), data[s:s + int(w) * int(h) * 4]) for s, (w, h) in zip(starts, sizes)]


def _glyphs(rng, n, box, lo, hi):
    """n closed outlines of lo-hi cubics that wander around an ellipse, concatenated."""
    k = rng.integers(lo, hi + 1, n)
    count = k + 3
    off = np.concatenate([[0], np.cumsum(count)[:-1]])
    nodes = np.zeros(int(count.sum()), NODE_DTYPE)
    for i in range(n):
        m = int(k[i])
        t = np.sort(rng.uniform(0.0, 2 * math.pi, m))
        r = box * rng.uniform(0.25, 0.45, 2)
        wob = rng.uniform(0.6, 1.0, m)
        ends = np.stack([box / 2 + r[0] * wob * np.cos(t), box / 2 + r[1] * wob * np.sin(t)], 1)
        prev = np.roll(ends, 1, 0)
        c1 = np.clip(prev + rng.uniform(-box / 8, box / 8, (m, 2)), 0, box)
        c2 = np.clip(ends + rng.uniform(-box / 8, box / 8, (m, 2)), 0, box)
        nd = nodes[off[i]:off[i] + count[i]]
        nd["tag"] = abi.CURVE_TO
        nd["p"][1:m + 1] = np.concatenate([c1, c2, ends], 1)
        nd["tag"][0] = nd["tag"][m + 2] = abi.MOVE_TO
        nd["p"][[0, m + 2], :2] = ends[-1]
        nd["tag"][m + 1] = abi.CLOSE_PATH
    return nodes, off, count


# ------------------------------------------------------------------ states
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "star":
        w, h, nodes, pattern, opts = star_300()
        # another seed's star is turned and coloured otherwise
        a = 0.1 * (seed % 63)
        c, s = math.cos(a), math.sin(a)
        for nd in nodes:
            if nd["tag"] != abi.CLOSE_PATH:
                x, y = nd["p"][0] - 150.0, nd["p"][1] - 150.0
                nd["p"][:2] = 150.0 + c * x - s * y, 150.0 + s * x + c * y
        st |= {"surface": _surface(seed, case["format"], w, h), "nodes": nodes, "pattern": _source(rng, "pixel", nodes),
               "opts": opts}
    elif kind == "fill":
        nodes = _one_path(rng, case)
        st |= {"surface": _surface(seed, case["format"], case["w"], case["h"]), "nodes": nodes,
               "pattern": _source(rng, case["source"], nodes),
               "opts": FillOptions(anti_aliasing=case["aa"], fill_rule="even_odd")}
    elif kind == "stroke":
        nodes = _one_path(rng, case)[:-2]  # an open path
        st |= {"surface": _surface(seed, case["format"], case["w"], case["h"]), "nodes": nodes,
               "pattern": _source(rng, "pixel", nodes),
               "opts": StrokeOptions(line_width=case["width"], line_join=case["join"], line_cap=case["cap"],
                                     dashes=_dashes(rng) if case["dashed"] else ())}
    elif kind == "batch":
        nodes, off, cnt = random_path_batch(rng, case["n"], case["w"], case["h"], case["side_lo"], case["side_hi"], 3,
                                            case["seg_hi"])
        st |= {"surface": _surface(seed, case["format"], case["w"], case["h"]), "nodes": nodes, "keep": []}
        cmds = (abi.z2d_fill_cmd * case["n"])()
        for i in range(case["n"]):
            p = _source(rng, case["source"], nodes[off[i]:off[i] + cnt[i]]).to_abi(st["keep"])
            cmds[i].pattern = C.pointer(p)
            cmds[i].node_offset, cmds[i].n_nodes = int(off[i]), int(cnt[i])
            cmds[i].opts = FillOptions(anti_aliasing=case["aa"], fill_rule=("even_odd", "non_zero")[i % 2],
                                       operator=case["op"]).to_abi()
        st["cmds"] = cmds
    elif kind == "jobs":
        sizes = _job_sizes(case)
        st["data"], surfaces = _atlas(seed, sizes)
        parts, base, ncmd, first, count = [], 0, 0, [], []
        for w, h in sizes:
            n, s = int(rng.integers(1, case["paths_hi"] + 1)), min(w, h)
            nodes, off, cnt = random_path_batch(rng, n, int(w), int(h), max(2.0, s / 64), max(4.0, s / 2))
            parts.append((nodes, off + base, cnt))
            first.append(ncmd)
            count.append(n)
            base, ncmd = base + len(nodes), ncmd + n
        nodes, off, cnt = (np.concatenate([p[k] for p in parts]) for k in range(3))
        stroke = rng.random(ncmd) < case["strokes"]
        dashed = stroke & (rng.random(ncmd) < 0.5)
        st["batch"] = PackedDrawBatch(nodes, off, cnt, _colours(rng, ncmd), np.arange(ncmd) % 2, stroke,
                                      rng.uniform(0.5, 20.0, ncmd), rng.integers(0, 3, ncmd), rng.integers(0, 3, ncmd),
                                      [_dashes(rng) if d else () for d in dashed])
        st["batch"].set_jobs(surfaces, first, count)
    elif kind == "glyphs":
        n, box = case["n"], case["box"]
        st["data"], surfaces = _atlas(seed, [(box, box)] * n)
        nodes, off, cnt = _glyphs(rng, n, float(box), case["cubics_lo"], case["cubics_hi"])
        st["batch"] = PackedBatch(nodes, off, cnt, _colours(rng, n), np.full(n, abi.FILL_NON_ZERO))
        st["batch"].set_jobs(surfaces, np.arange(n), np.ones(n, int))
    elif kind == "mask":
        w, h = case["w"], case["h"]
        if case["source"] == "pixel":
            src = _source(rng, "pixel", None)
        else:
            g = _gradient(rng, case["source"], case["method"], w * 0.02, h * 0.03, w * 0.97, h * 0.9, 4)
            src = Pattern.from_gradient(g) if case["dither"] == "none" else Pattern.dither(case["dither"], g, 8)
        mask = _surface(seed + 1, "alpha8", w, h)
        st |= {"surface": _surface(seed, case["format"], w, h), "precision": case["precision"],
               "ops": [Operation("dst_in", dst=src, src=mask), Operation(case["op"])]}
    elif kind == "layer":
        st |= {"surface": _surface(seed, case["format"], case["w"], case["h"]), "op": case["op"], "x": case["x"],
               "y": case["y"], "layer": _surface(seed + 1, case["format"], case["sw"], case["sh"])}
    else:  # a drawing with a plain ground
        w, h = case["w"], case["h"]
        s = Surface(case["format"], w, h)
        s.paint_pixel(Pixel.rgba(*map(int, _colours(rng, 1)[0])))
        s = s.to_device()
        nodes, off, cnt = random_path_batch(rng, 60, w, h, 4.0, max(8.0, min(w, h) / 2))
        PackedBatch(nodes, off, cnt, _colours(rng, 60), np.arange(60) % 2).fill_batch(s)
        st |= {"surface": s, "profile": None if case["profile"] == "none" else case["profile"]}
    return st


def run(st):
    kind = st["kind"]
    if kind in ("star", "fill"):
        painter.fill(st["surface"], st["pattern"], st["nodes"], st["opts"])
    elif kind == "stroke":
        painter.stroke(st["surface"], st["pattern"], st["nodes"], st["opts"])
    elif kind == "batch":
        painter.fill_batch_arrays(st["surface"], st["nodes"], st["cmds"])
    elif kind == "jobs":
        st["batch"].draw_jobs()
        return st["data"]
    elif kind == "glyphs":
        st["batch"].fill_jobs()
        return st["data"]
    elif kind == "mask":
        compositor.SurfaceCompositor.run(st["surface"], 0, 0, st["ops"], st["precision"])
    elif kind == "layer":
        compositor.composite(st["surface"], st["layer"], st["op"], st["x"], st["y"])
    else:
        return np.frombuffer(png.scanlines(st["surface"], st["profile"]), np.uint8)
    return st["surface"].data
