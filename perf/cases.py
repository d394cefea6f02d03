"""The work a user of this library has it do, as measurable cases.

Each case goes through the public entry points (Plotter, fill_batch, PreparedBatch,
composite_batch, Adjoint, StrokeComposite, Context.convert) with one Context kept for the
whole program on one torch stream, as a program that draws frame after frame keeps it.

Kinds of case:
  path       one Plotter.fill / Plotter.stroke call on a device raster
  batch      many independent fills or strokes: a PreparedBatch replayed, a fill_batch call on
             device buffers, or a fill_batch call on pinned host buffers
  composite  an ordered sequence of calls on one canvas (composite_batch)
  adjoint    differentiable coverage of a batch and its gradients (Adjoint)
  paint      the differentiable ordered composite of strokes and its gradients
             (StrokeComposite)
  convert    a drawn raster to straight sRGB (Context.convert)
"""
import math

import numpy as np
import torch

from footile_gb300 import _abi
from footile_gb300._lib import Context
from footile_gb300.adjoint import Adjoint, StrokeComposite
from footile_gb300.path import FillRule, JoinStyle
from footile_gb300.plotter import Plotter, PreparedBatch, composite_batch, fill_batch

JOINS = {"miter": JoinStyle.Miter(4.0), "bevel": JoinStyle.Bevel, "round": JoinStyle.Round}
GLYPH_MIX = (0.7, 0.2, 0.1)  # quads, cubics, lines: outlines of a font
EVEN_MIX = (1 / 3, 1 / 3, 1 / 3)
CUBICS = (0.0, 1.0, 0.0)


# ------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: one closed 64-segment path on a 256 x 256 mask
        {"name": "path_256", "kind": "path", "w": 256, "h": 256, "subs": 1, "segs": 64, "extent": 1.0, "rgba": False,
         "evenodd": False, "pen": 0.0, "join": "miter"},
        # one small drawn line of a user interface: an open curve stroked on a ragged canvas
        {"name": "pen_97x61", "kind": "path", "w": 97, "h": 61, "subs": 1, "segs": 12, "extent": 1.0, "rgba": True,
         "evenodd": False, "pen": 3.0, "join": "bevel"},
        # a page of vector art: many shapes of one path on an odd-sized colour canvas
        {"name": "poster_1531x1117", "kind": "path", "w": 1531, "h": 1117, "subs": 90, "segs": 40, "extent": 0.2,
         "rgba": True, "evenodd": True, "pen": 0.0, "join": "miter"},
        # the large self-intersecting scene: 1,000 sub-paths of 100 segments, filled and stroked
        {"name": "scene_4096", "kind": "path", "w": 4096, "h": 4096, "subs": 1000, "segs": 100, "extent": 1.0,
         "rgba": False, "evenodd": False, "pen": 0.0, "join": "miter"},
        {"name": "scene_4096_stroke", "kind": "path", "w": 4096, "h": 4096, "subs": 1000, "segs": 100, "extent": 1.0,
         "rgba": True, "evenodd": False, "pen": 8.0, "join": "round"},
        # a glyph atlas: 65,536 uneven paths, planned once and replayed
        {"name": "glyphs_65536", "kind": "batch", "paths": 65536, "min_seg": 4, "max_seg": 400, "min_side": 16,
         "max_side": 256, "rgba": False, "evenodd": False, "pen": 0.0, "how": "prepared"},
        # a page of text in colour: new glyphs with every call
        {"name": "text_3000_rgba", "kind": "batch", "paths": 3000, "min_seg": 4, "max_seg": 120, "min_side": 12,
         "max_side": 96, "rgba": True, "evenodd": True, "pen": 0.0, "how": "call"},
        # glyphs for a program whose masks live in page-locked host memory
        {"name": "glyphs_host_16384", "kind": "batch", "paths": 16384, "min_seg": 4, "max_seg": 400, "min_side": 16,
         "max_side": 256, "rgba": False, "evenodd": False, "pen": 0.0, "how": "host"},
        # a drawing of many strokes, composited in order on one canvas
        {"name": "strokes_16384", "kind": "composite", "paths": 16384, "w": 2048, "h": 2048, "min_seg": 8,
         "max_seg": 64, "rgba": True, "pen": 12.0, "join": "miter"},
        # fitting curves to images: coverage of 1,024 closed cubic paths and its gradients
        {"name": "fit_1024", "kind": "adjoint", "paths": 1024, "side": 128, "segs": 32, "evenodd": False, "pen": 0.0},
        # fitting an ordered painting of strokes, gradients to control points and widths
        {"name": "paint_400_480x360", "kind": "paint", "paths": 400, "w": 480, "h": 360, "min_seg": 8, "max_seg": 64,
         "pen": 12.0},
        # a finished drawing to sRGB for display
        {"name": "convert_8192", "kind": "convert", "w": 8192, "h": 8192, "rgba": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["path", "path", "path", "batch", "batch", "batch", "composite", "adjoint", "paint", "convert"])
    rgba, evenodd = rng.random() < 0.5, rng.random() < 0.5
    join = rng.choice(sorted(JOINS))
    if kind == "path":
        w, subs = _log(rng, 40, 4096), _log(rng, 1, 1000)
        pen = round(rng.uniform(1.0, 12.0), 2) if rng.random() < 0.4 else 0.0
        extent = 1.0 if rng.random() < 0.4 else round(rng.uniform(0.05, 0.5), 3)
        # small canvases hold small drawings
        subs = max(1, min(subs, w * w // 4000))
        return {"kind": kind, "w": w, "h": max(16, int(w * rng.uniform(0.4, 1.6)) | 1), "subs": subs,
                "segs": _log(rng, 4, 100), "extent": extent, "rgba": rgba, "evenodd": evenodd and not pen, "pen": pen,
                "join": join}
    if kind == "batch":
        lo = _log(rng, 10, 40)
        how = rng.choice(["prepared", "call", "host"])
        pen = round(rng.uniform(1.0, 6.0), 2) if rng.random() < 0.2 else 0.0
        top = 16384 if how == "host" else (8192 if pen else 65536)
        return {"kind": kind, "paths": _log(rng, 300, top), "min_seg": 4, "max_seg": _log(rng, 20, 200 if pen else 400),
                "min_side": lo, "max_side": _log(rng, lo + 8, 256), "rgba": rgba and how != "host",
                "evenodd": evenodd and not pen, "pen": pen, "how": how}
    if kind == "composite":
        return {"kind": kind, "paths": _log(rng, 200, 8000), "w": _log(rng, 300, 2048), "h": _log(rng, 300, 2048),
                "min_seg": 4, "max_seg": _log(rng, 8, 64), "rgba": rng.random() < 0.8,
                "pen": round(rng.uniform(2.0, 12.0), 2), "join": join}
    if kind == "adjoint":
        pen = round(rng.uniform(2.0, 12.0), 2) if rng.random() < 0.4 else 0.0
        return {"kind": kind, "paths": _log(rng, 16, 200 if pen else 1024), "side": _log(rng, 33, 192),
                "segs": _log(rng, 4, 32), "evenodd": evenodd and not pen, "pen": pen}
    if kind == "paint":
        return {"kind": kind, "paths": _log(rng, 16, 400), "w": _log(rng, 60, 480), "h": _log(rng, 60, 400),
                "min_seg": 4, "max_seg": _log(rng, 8, 64), "pen": round(rng.uniform(2.0, 12.0), 2)}
    return {"kind": "convert", "w": _log(rng, 200, 8192), "h": _log(rng, 200, 8192), "rgba": rgba}


# ----------------------------------------------------------------------- inputs
def _paths_ops(rng, n_seg, box, mix, close, widths=None):
    """Op records of len(n_seg) sub-paths: [PenWidth], Move, n_seg segments, [Close].
    `box`: (n, 4) x, y, width, height of the rectangle each sub-path's points lie in.
    Returns (ops, first op and op count of every sub-path)."""
    n_seg = np.asarray(n_seg, np.int64)
    n, lead = len(n_seg), 1 if widths is not None else 0
    per = n_seg + 1 + lead + (1 if close else 0)
    begin = np.cumsum(per) - per
    ops = np.zeros(int(per.sum()), _abi.OP_DTYPE)
    box = box.astype(np.float32)
    if widths is not None:
        ops["kind"][begin] = _abi.OP_PEN_WIDTH
        ops["v"][begin, 0] = widths
    ops["kind"][begin + lead] = _abi.OP_MOVE
    ops["v"][begin + lead, 0:2] = box[:, 0:2] + rng.random((n, 2), np.float32) * box[:, 2:4]
    at = np.repeat(begin + lead + 1, n_seg) + (np.arange(int(n_seg.sum())) - np.repeat(np.cumsum(n_seg) - n_seg, n_seg))
    of = np.repeat(np.arange(n), n_seg)
    u = rng.random(len(at))
    kind = np.where(u < mix[0], _abi.OP_QUAD, np.where(u < mix[0] + mix[1], _abi.OP_CUBIC, _abi.OP_LINE))
    v = np.tile(box[of, 0:2], 3) + rng.random((len(at), 6), np.float32) * np.tile(box[of, 2:4], 3)
    v[kind == _abi.OP_LINE, 2:] = 0
    v[kind == _abi.OP_QUAD, 4:] = 0
    ops["kind"][at] = kind
    ops["v"][at] = v
    if close:
        ops["kind"][begin + per - 1] = _abi.OP_CLOSE
    return ops, begin, per


def _rects(rng, n, w, h, extent):
    ext = extent * rng.uniform(0.5, 1.0, (n, 2)) if extent < 1.0 else np.ones((n, 2))
    size = ext * [w, h]
    return np.concatenate([rng.random((n, 2)) * ([w, h] - size), size], 1)


def _clrs(rng, n):
    rgb, alpha = rng.integers(0, 256, (n, 3)), rng.integers(64, 256, n)
    clr = np.zeros((n, 4), np.uint8)
    clr[:, :3] = (rgb * alpha[:, None] + 127) // 255
    clr[:, 3] = alpha
    return clr


def _descs(begin, per, w, h, stride, offset):
    paths = np.zeros(len(begin), _abi.PATH_DTYPE)
    paths["op_begin"], paths["n_ops"] = begin, per
    paths["width"], paths["height"], paths["stride"], paths["raster_offset"] = w, h, stride, offset
    paths["s_width"] = 1.0
    return paths


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).cuda()


_kept = []


def _sizes(c, rng):
    """Segment counts and canvas sides (log-uniform; 0 without canvases of their own) of a
    case's paths: the same set for every seed, in an order of its own."""
    own, n = np.random.default_rng([c["paths"], c["min_seg"], c["max_seg"]]), c["paths"]

    def spread(lo, hi):
        return np.rint(np.exp(own.uniform(math.log(lo), math.log(hi), n))).astype(np.int64)

    order = rng.permutation(n)
    if "min_side" in c:
        return spread(c["min_seg"], c["max_seg"])[order], spread(c["min_side"], c["max_side"])[order]
    return own.integers(c["min_seg"], c["max_seg"] + 1, n)[order], 0


def _context():
    """The program's Context, on the torch stream that the program works on."""
    if not _kept:
        stream = torch.cuda.Stream()
        torch.cuda.set_stream(stream)
        ctx = Context(0)
        ctx.set_stream(stream.cuda_stream)
        _kept.extend([ctx, stream])
    return _kept[0]


def _path_case(c, rng):
    subs = np.full(c["subs"], c["segs"])
    ops, _, _ = _paths_ops(rng, subs, _rects(rng, c["subs"], c["w"], c["h"], c["extent"]), EVEN_MIX, not c["pen"],
                           np.full(c["subs"], c["pen"], np.float32) if c["pen"] else None)
    return ops


def _batch_case(c, rng):
    n = c["paths"]
    segs, side = _sizes(c, rng)
    box = np.zeros((n, 4))
    box[:, 2] = box[:, 3] = side
    ops, begin, per = _paths_ops(rng, segs, box, GLYPH_MIX, True,
                                 np.full(n, c["pen"], np.float32) if c["pen"] else None)
    stride = side * 4 if c["rgba"] else (side + 3) // 4 * 4
    size = stride * side
    paths = _descs(begin, per, side, side, stride, np.cumsum(size) - size)
    paths["clr"] = _clrs(rng, n)
    return ops, paths, int(size.sum())


def _strokes(c, rng, w, h):
    n = c["paths"]
    segs, _ = _sizes(c, rng)
    return _paths_ops(rng, segs, np.tile([0.0, 0.0, w, h], (n, 1)), CUBICS, False,
                      rng.uniform(1.0, c["pen"], n).astype(np.float32))


def _adjoint_case(c, rng):
    n, s = c["paths"], c["side"]
    # clear of the canvas edges, as in the repository's own gradient batch
    m = s / 8
    ops, begin, per = _paths_ops(rng, np.full(n, c["segs"]), np.tile([m, m, s - 2 * m, s - 2 * m], (n, 1)), CUBICS,
                                 not c["pen"], rng.uniform(1.0, c["pen"], n).astype(np.float32) if c["pen"] else None)
    paths = _descs(begin, per, s, s, 4 * s, np.arange(n) * 4 * s * s)
    return ops, paths, rng.random(n * s * s, np.float32)


def _paint_case(c, rng):
    w, h = c["w"], c["h"]
    m = min(w, h) / 16
    n = c["paths"]
    segs, _ = _sizes(c, rng)
    ops, begin, per = _paths_ops(rng, segs, np.tile([m, m, w - 2 * m, h - 2 * m], (n, 1)), CUBICS, False,
                                 rng.uniform(1.0, c["pen"], n).astype(np.float32))
    clr = _clrs(rng, n).astype(np.float32) / 255
    return ops, _descs(begin, per, w, h, 4 * w, 0), clr, rng.random((w * h, 4), np.float32)


def prepare(case, seed):
    c, rng, ctx = case, np.random.default_rng(seed), _context()
    kind = c["kind"]
    if kind == "path":
        ops = _path_case(c, rng)
        shape = (c["h"], c["w"], 4) if c["rgba"] else (c["h"], c["w"])
        raster = torch.zeros(shape, dtype=torch.uint8, device="cuda")
        return {"kind": kind, "plotter": Plotter(raster, context=ctx), "ops": _dev(ops), "rule": FillRule(int(c["evenodd"])),
                "clr": tuple(int(v) for v in _clrs(rng, 1)[0]), "stroke": bool(c["pen"]), "join": JOINS[c["join"]]}
    if kind == "batch":
        ops, paths, nbytes = _batch_case(c, rng)
        fmt, rule, stroke = _abi.RGBA8P if c["rgba"] else _abi.MATTE8, int(c["evenodd"]), bool(c["pen"])
        s = {"kind": c["how"], "ctx": ctx, "paths": paths, "fmt": fmt, "rule": rule, "stroke": stroke}
        if c["how"] == "host":
            pin = torch.from_numpy(ops.view(np.uint8)).pin_memory()
            ras = torch.zeros(nbytes, dtype=torch.uint8).pin_memory()
            return s | {"keep": (pin, ras), "ops": pin.numpy().view(_abi.OP_DTYPE), "raster": ras.numpy()}
        s |= {"ops": _dev(ops), "raster": torch.zeros(nbytes, dtype=torch.uint8, device="cuda")}
        if c["how"] == "prepared":
            s["batch"] = PreparedBatch(ctx, paths, fmt, rule, stroke)
        return s
    if kind == "composite":
        ops, begin, per = _strokes(c, rng, c["w"], c["h"])
        paths = _descs(begin, per, c["w"], c["h"], c["w"] * (4 if c["rgba"] else 1), 0)
        paths["clr"] = _clrs(rng, c["paths"])
        shape = (c["h"], c["w"], 4) if c["rgba"] else (c["h"], c["w"])
        return {"kind": kind, "ctx": ctx, "ops": _dev(ops), "paths": paths, "fmt": _abi.RGBA8P if c["rgba"] else _abi.MATTE8,
                "raster": torch.zeros(shape, dtype=torch.uint8, device="cuda"), "join": JOINS[c["join"]]}
    if kind == "adjoint":
        ops, paths, target = _adjoint_case(c, rng)
        n = len(target)
        return {"kind": kind, "adj": Adjoint(ctx), "ctx": ctx, "ops": _dev(ops), "paths": paths, "rule": int(c["evenodd"]),
                "stroke": bool(c["pen"]), "target": torch.from_numpy(target).cuda(),
                "cov": torch.empty(n, device="cuda"), "g_ops": torch.empty((len(ops), 6), device="cuda"),
                "g_width": torch.empty(len(paths), device="cuda")}
    if kind == "paint":
        ops, paths, clr, target = _paint_case(c, rng)
        return {"kind": kind, "comp": StrokeComposite(ctx), "ctx": ctx, "ops": _dev(ops), "paths": paths, "w": c["w"],
                "h": c["h"], "clr": torch.from_numpy(clr).cuda(), "target": torch.from_numpy(target).cuda(),
                "out": torch.empty((c["w"] * c["h"], 4), device="cuda"),
                "g_ops": torch.empty((len(ops), 6), device="cuda"), "g_width": torch.empty(len(paths), device="cuda")}
    # a drawing: flat areas of a few colours, soft edges, an empty background
    h, w = c["h"], c["w"]
    src = torch.zeros((h, w, 4) if c["rgba"] else (h, w), dtype=torch.uint8, device="cuda")
    ops, _, _ = _paths_ops(rng, np.full(60, 24), _rects(rng, 60, w, h, 0.5), EVEN_MIX, True)
    for k, clr in enumerate(_clrs(rng, 6)):
        part = ops[k * len(ops) // 6:(k + 1) * len(ops) // 6]
        Plotter(src, context=ctx).fill(FillRule.NonZero, _dev(part), tuple(int(v) for v in clr))
        torch.cuda.synchronize()
    return {"kind": kind, "ctx": ctx, "src": src, "dst": torch.empty_like(src)}


# ------------------------------------------------------------------------- runs
def run(s):
    kind = s["kind"]
    if kind == "path":
        if s["stroke"]:
            return s["plotter"].set_join(s["join"]).stroke(s["ops"], s["clr"])
        return s["plotter"].fill(s["rule"], s["ops"], s["clr"])
    if kind == "prepared":
        if s["stroke"]:
            s["ctx"].set_join(JOINS["miter"].kind, JOINS["miter"].limit)
        s["batch"].launch(s["ops"], s["raster"])
        return s["raster"]
    if kind in ("call", "host"):
        if s["stroke"]:
            s["ctx"].set_join(JOINS["miter"].kind, JOINS["miter"].limit)
        status = fill_batch(s["ctx"], s["ops"], s["paths"], s["fmt"], s["raster"], s["rule"], s["stroke"])
        return [s["raster"], status]
    if kind == "composite":
        s["ctx"].set_join(s["join"].kind, s["join"].limit)
        status = composite_batch(s["ctx"], s["ops"], s["paths"], s["fmt"], s["raster"], FillRule.NonZero, True)
        return [s["raster"], status]
    if kind == "adjoint":
        s["ctx"].set_join(JOINS["miter"].kind, JOINS["miter"].limit)
        cov = s["adj"].forward(s["rule"], s["ops"], s["paths"], s["cov"], s["stroke"])
        s["adj"].backward(2 * (cov - s["target"]), s["g_ops"], s["g_width"])
        return {"cov": cov, "g_ops": s["g_ops"], "g_width": s["g_width"]}
    if kind == "paint":
        s["ctx"].set_join(JOINS["miter"].kind, JOINS["miter"].limit)
        out = s["comp"].forward(s["ops"], s["paths"], s["clr"], s["w"], s["h"], s["out"])
        s["comp"].backward(2 * (out - s["target"]), s["g_ops"], s["g_width"])
        return {"out": out, "g_ops": s["g_ops"], "g_width": s["g_width"]}
    return s["ctx"].convert(s["src"], s["dst"])


# ------------------------------------------------------------------------- work
def work(case):
    """Bytes: ops, descriptors and inputs read once, outputs written once (Rgba8p canvases
    are read and written).  Flops only where floats are accumulated per pixel and layer."""
    c, kind = case, case["kind"]
    if kind == "path":
        px = c["w"] * c["h"]
        return {"bytes": 32 * c["subs"] * (c["segs"] + 2) + px * (8 if c["rgba"] else 1), "flops": 0}
    if kind == "batch":
        def mean_of(lo, hi, p):  # of x^p, x log-uniform in [lo, hi]
            return (hi ** p - lo ** p) / (p * math.log(hi / lo))
        px = c["paths"] * mean_of(c["min_side"], c["max_side"], 2)
        ops = c["paths"] * (mean_of(c["min_seg"], c["max_seg"], 1) + 2)
        return {"bytes": 32 * ops + 40 * c["paths"] + px * (8 if c["rgba"] else 1), "flops": 0}
    if kind == "convert":
        return {"bytes": 2 * c["w"] * c["h"] * (4 if c["rgba"] else 1), "flops": 0}
    if kind == "adjoint":
        ops, px = c["paths"] * (c["segs"] + 2), c["paths"] * c["side"] ** 2
        return {"bytes": (32 + 24) * ops + 8 * px, "flops": 8 * px}
    ops, px = c["paths"] * ((c["min_seg"] + c["max_seg"]) / 2 + 2), c["w"] * c["h"]
    if kind == "paint":
        return {"bytes": (32 + 24) * ops + 16 * 4 * px, "flops": 20 * c["paths"] * px}
    return {"bytes": 32 * ops + 40 * c["paths"] + px * (8 if c["rgba"] else 1), "flops": 0}


# ------------------------------------------------------------------------ exact
# Coverage and gradients in 64 bits: the curves' subdivision and the joins' kinds are
# decided in float32 as the path does (they are discrete), everything else is float64.
def _mid(a, b):
    return ((a + b).astype(np.float32) * np.float32(0.5)).astype(np.float32)


def _flatten(ctrl, tol_sq):
    """Leaves of every cubic (n, 4, 2) f32: (cubic, end parameter, end point f32), in order."""
    cub, t0, h = np.arange(len(ctrl)), np.zeros(len(ctrl)), np.ones(len(ctrl))
    a, b, c, d = (ctrl[:, k].astype(np.float32) for k in range(4))
    done = []
    while len(cub):
        ab, bc, cd = _mid(a, b), _mid(b, c), _mid(c, d)
        abc, bcd = _mid(ab, bc), _mid(bc, cd)
        m = _mid(abc, bcd)
        e = (m - _mid(a, d)).astype(np.float32)
        sq = (e * e).astype(np.float32)
        flat = (sq[:, 0] + sq[:, 1]).astype(np.float32) <= tol_sq
        done.append((cub[flat], t0[flat] + h[flat], d[flat]))
        k = ~flat
        cub, t0, h = np.tile(cub[k], 2), np.concatenate([t0[k], t0[k] + h[k] / 2]), np.tile(h[k] / 2, 2)
        a, b, c, d = (np.concatenate(p) for p in ((a[k], m[k]), (ab[k], bcd[k]), (abc[k], cd[k]), (m[k], d[k])))
    cub, t, p = (np.concatenate(x) for x in zip(*done))
    order = np.lexsort((t, cub))
    return cub[order], t[order], p[order]


def _bernstein(ctrl, cub, t):
    t = torch.from_numpy(t)[:, None]
    u, k = 1 - t, ctrl[torch.from_numpy(cub)]
    return u ** 3 * k[:, 0] + 3 * t * u ** 2 * k[:, 1] + 3 * t ** 2 * u * k[:, 2] + t ** 3 * k[:, 3]


def _fixed(p):
    return np.trunc(p.astype(np.float64) * 65536).astype(np.int64)


def _direction(p, first, count):
    """+1 / -1 per polygon: the turn at its first top vertex, in 16.16."""
    sign = np.ones(len(first))
    q = _fixed(p)
    for i, (f, n) in enumerate(zip(first, count)):
        v = q[f:f + n]
        v = v[np.concatenate([[True], (v[1:] != v[:-1]).any(1)])] if n else v
        if len(v) > 1 and (v[0] == v[-1]).all():
            v = v[:-1]
        if len(v) < 2:
            continue
        k = np.lexsort((np.arange(len(v)), v[:, 0], v[:, 1]))[0]
        a, b = v[k - 1] - v[k], v[(k + 1) % len(v)] - v[k]
        sign[i] = 1.0 if (a[0] * b[1] >> 16) > (b[0] * a[1] >> 16) else -1.0
    return sign


def _pieces(p0, p1, w, h):
    """Every edge cut at pixel borders: (edge, row, cell, height, mid x, from, to), `from`
    and `to` along the edge from p0; cell -1 is left of the canvas."""
    down = p1[:, 1] > p0[:, 1]
    a, b = np.where(down[:, None], p0, p1), np.where(down[:, None], p1, p0)
    r0 = np.clip(np.floor(a[:, 1]), 0, None).astype(np.int64)
    r1 = np.clip(np.ceil(b[:, 1]) - 1, None, h - 1).astype(np.int64)
    n = np.where(a[:, 1] < b[:, 1], np.maximum(r1 - r0 + 1, 0), 0)
    e = np.repeat(np.arange(len(p0)), n)
    r = np.repeat(r0 - (np.cumsum(n) - n), n) + np.arange(len(e))
    ax, ay, dy = a[e, 0], a[e, 1], (b[:, 1] - a[:, 1])[e]
    slope = (b[e, 0] - ax) / dy
    yt, yb = np.maximum(ay, r), np.minimum(b[e, 1], r + 1.0)
    xt, xb = ax + (yt - ay) * slope, ax + (yb - ay) * slope
    ut, ub = (yt - ay) / dy, (yb - ay) / dy
    xl, xr = np.minimum(xt, xb), np.maximum(xt, xb)
    c0 = np.maximum(np.floor(xl), -1).astype(np.int64)
    c1 = np.clip(np.floor(xr), -1, w - 1).astype(np.int64)
    n = np.maximum(c1 - c0 + 1, 0)
    i = np.repeat(np.arange(len(e)), n)
    c = np.repeat(c0 - (np.cumsum(n) - n), n) + np.arange(len(i))
    lo, hi = np.where(c < 0, xl[i], np.maximum(xl[i], c)), np.minimum(xr[i], c + 1.0)
    span = xr[i] - xl[i]
    flat = span <= 0
    f0, f1 = np.where(flat, 0.0, (lo - xl[i]) / np.where(flat, 1, span)), np.where(flat, 1.0, (hi - xl[i]) / np.where(flat, 1, span))
    rising = (xt <= xb)[i]
    du = (ub - ut)[i]
    u0, u1 = np.where(rising, ut[i] + f0 * du, ub[i] - f1 * du), np.where(rising, ut[i] + f1 * du, ub[i] - f0 * du)
    ei, d = e[i], down[e[i]]
    return ei, r[i], c, (f1 - f0) * (yb - yt)[i] * np.where(d, 1.0, -1.0), (lo + hi) / 2, np.where(d, u0, 1 - u1), np.where(d, u1, 1 - u0)


class _Cover(torch.autograd.Function):
    """Coverage planes of closed polygons (vertices f64, polygon i on plane i)."""

    @staticmethod
    def forward(ctx, verts, nxt, plane, sign, n, w, h, evenodd):
        v = verts.detach().numpy()
        ei, r, c, dh, xm, u0, u1 = _pieces(v, v[nxt], w, h)
        base = (plane[ei] * h + r) * w
        left = c < 0
        s = np.bincount(base + np.maximum(c, 0), np.where(left, dh, dh * (c + 1 - xm)), n * h * w)
        k = ~left & (c + 1 < w)
        s += np.bincount(base[k] + c[k] + 1, (dh * (xm - c))[k], n * h * w)
        s = np.cumsum(s.reshape(n, h, w), 2) * sign[:, None, None]
        if evenodd:
            m = s - 2 * np.floor(s / 2)
            cov, d = np.where(m <= 1, m, 2 - m), np.where(m < 1, 1.0, -1.0)
        else:
            cov, d = np.clip(s, 0, 1), ((s > 0) & (s < 1)).astype(np.float64)
        k = ~left
        ctx.saved = (v, nxt, ei[k], (base + c)[k], u0[k], u1[k], (d * sign[:, None, None]).reshape(-1))
        return torch.from_numpy(cov.reshape(-1))

    @staticmethod
    def backward(ctx, grad):
        v, nxt, ei, at, u0, u1, d = ctx.saved
        g = grad.numpy()[at] * d[at]
        whole, later = u1 - u0, (u1 * u1 - u0 * u0) / 2
        e = v[nxt] - v
        perp = np.stack([-e[:, 1], e[:, 0]], 1)
        ga, gb = np.bincount(ei, g * (whole - later), len(v)), np.bincount(ei, g * later, len(v))
        out = ga[:, None] * perp
        np.add.at(out, nxt, gb[:, None] * perp)
        return (torch.from_numpy(out),) + (None,) * 7


def _cubics(ops, paths, pens):
    """Control points (n, 4, 2) f64 of a batch of cubic paths, where they come from in
    the op floats, and the path of each."""
    is_c = ops["kind"] == _abi.OP_CUBIC
    at = np.flatnonzero(is_c)
    v = torch.from_numpy(ops["v"].astype(np.float64)).requires_grad_(True)
    prev = at - 1
    pen = torch.where(torch.from_numpy(is_c[prev])[:, None], v[prev, 4:6], v[prev, 0:2])
    ctrl = torch.stack([pen, v[at, 0:2], v[at, 2:4], v[at, 4:6]], 1)
    path = np.searchsorted(paths["op_begin"], at, "right") - 1
    return v, ctrl, path


def _ring(first, count):
    nxt = np.arange(int(count.sum())) + 1
    nxt[first + count - 1] = first
    return nxt


def _fills(ops, paths):
    v, ctrl, path = _cubics(ops, paths, 0)
    cub, t, p32 = _flatten(ctrl.detach().numpy(), np.float32(0.3) * np.float32(0.3))
    starts = torch.from_numpy(paths["op_begin"].astype(np.int64))
    move = v[starts, 0:2]
    verts, own = _bernstein(ctrl, cub, t), path[cub]
    n = len(paths)
    order = np.argsort(np.concatenate([np.arange(n) * 2, own * 2 + 1]), kind="stable")
    verts = torch.cat([move, verts])[torch.from_numpy(order)]
    p32 = np.concatenate([move.detach().numpy().astype(np.float32), p32])[order]
    count = np.bincount(own, minlength=n) + 1
    first = np.cumsum(count) - count
    return v, verts, _ring(first, count), np.repeat(np.arange(n), count), _direction(p32, first, count)


def _norm32(d):
    sq = (d * d).astype(np.float32)
    return (d / np.sqrt((sq[:, 0] + sq[:, 1]).astype(np.float32)).astype(np.float32)[:, None]).astype(np.float32)


def _cross(a0, a1, b0, b1, stack):
    """Intersection of the lines a0-a1 and b0-b1, and the determinant."""
    x1, y1, x2, y2, x3, y3, x4, y4 = (q for p in (a0, a1, b0, b1) for q in (p[:, 0], p[:, 1]))
    den = (x1 - x2) * (y3 - y4) - (y1 - y2) * (x3 - x4)
    a, b = x1 * y2 - y1 * x2, x3 * y4 - y3 * x4
    return stack([(a * (x3 - x4) - (x1 - x2) * b) / den, (a * (y3 - y4) - (y1 - y2) * b) / den], 1), den


def _strokes_outline(ops, paths):
    """Outlines (miter limit 4) of open cubic strokes with one PenWidth op each."""
    v, ctrl, path = _cubics(ops, paths, 1)
    cub, t, p32 = _flatten(ctrl.detach().numpy(), np.float32(0.3) * np.float32(0.3))
    starts = torch.from_numpy(paths["op_begin"].astype(np.int64))
    move, width = v[starts + 1, 0:2], v[starts, 0]
    n = len(paths)
    own = path[cub]
    order = np.argsort(np.concatenate([np.arange(n) * 2, own * 2 + 1]), kind="stable")
    pts = torch.cat([move, _bernstein(ctrl, cub, t)])[torch.from_numpy(order)]
    p32 = np.concatenate([move.detach().numpy().astype(np.float32), p32])[order]
    own = np.concatenate([np.arange(n), own])[order]
    keep = np.concatenate([[True], (own[1:] != own[:-1]) | (p32[1:] != p32[:-1]).any(1)])
    pts, p32, own = pts[torch.from_numpy(np.flatnonzero(keep))], p32[keep], own[keep]
    # segments of both sides, in the order they are walked: forward, then back
    count = np.bincount(own, minlength=n)
    first = np.cumsum(count) - count
    seg = np.flatnonzero(own[1:] == own[:-1])
    back = np.concatenate([seg, -seg])
    order = np.lexsort((back, np.repeat([0, 1], len(seg)), np.tile(own[seg], 2)))
    i0, i1 = np.concatenate([seg, seg + 1])[order], np.concatenate([seg + 1, seg])[order]
    so, side = np.tile(own[seg], 2)[order], np.repeat([0, 1], len(seg))[order]

    def offsets(p, hw, norm, stack):
        d = p[i1] - p[i0]
        vr = norm(stack([d[:, 1], -d[:, 0]], 1)) * hw
        return p[i0] + vr, p[i1] + vr

    w32 = (width.detach().numpy().astype(np.float32) * np.float32(0.5))[so][:, None]
    a32, b32 = (x.astype(np.float32) for x in offsets(p32, w32, _norm32, np.stack))
    ts = torch.from_numpy(so)
    a64, b64 = offsets(pts, (width * 0.5)[ts][:, None], lambda d: d / d.norm(dim=1, keepdim=True), torch.stack)
    # joins between consecutive segments of one side, decided in float32
    j = np.flatnonzero((so[1:] == so[:-1]) & (side[1:] == side[:-1])) + 1
    u, q = (b32[j - 1] - a32[j - 1]).astype(np.float32), (a32[j] - b32[j]).astype(np.float32)

    def angle(d):
        return np.arctan2(d[:, 1].astype(np.float64), d[:, 0].astype(np.float64)).astype(np.float32)

    th, pi = (angle(u) - angle(q)).astype(np.float32), np.float32(np.pi)
    th = np.where(th < -pi, th + 2 * pi, np.where(th > pi, th - 2 * pi, th)).astype(np.float32)
    sm = np.abs(np.sin(th.astype(np.float64) / 2)).astype(np.float32)
    with np.errstate(all="ignore"):
        x32, den = _cross(a32[j - 1], b32[j - 1], a32[j], b32[j], np.stack)
    miter = (sm >= np.float32(0.25)) & (sm < 1) & (den != 0)
    jm, jb = j[miter], j[~miter]
    m64, _ = _cross(*(x[torch.from_numpy(k)] for x, k in ((a64, jm - 1), (b64, jm - 1), (a64, jm), (b64, jm))), torch.stack)
    heads = np.flatnonzero(np.concatenate([[True], (so[1:] != so[:-1]) | (side[1:] != side[:-1])]))
    tails = np.concatenate([heads[1:] - 1, [len(so) - 1]])
    parts = [(heads, 0, a64, a32, heads), (jm, 0, None, None, None), (jb, 0, b64, b32, jb - 1), (jb, 1, a64, a32, jb),
             (tails, 2, b64, b32, tails)]
    key = np.concatenate([4 * k + s for k, s, *_ in parts])
    order = np.argsort(key, kind="stable")
    verts = torch.cat([m64 if x is None else x[torch.from_numpy(at)] for _, _, x, _, at in parts])[torch.from_numpy(order)]
    v32 = np.concatenate([x32[miter] if x is None else x[at] for _, _, _, x, at in parts])[order]
    plane = np.concatenate([so[k] for k, *_ in parts])[order]
    count = np.bincount(plane, minlength=n)
    first = np.cumsum(count) - count
    return v, verts, _ring(first, count), plane, _direction(v32, first, count)


def exact(case, seed):
    """Coverage, composite and gradients in 64 bits; masks, rasters and conversions are
    whole numbers and have none."""
    c = case
    if c["kind"] not in ("adjoint", "paint"):
        return None
    rng = np.random.default_rng(seed)
    if c["kind"] == "adjoint":
        ops, paths, target = _adjoint_case(c, rng)
        w = h = c["side"]
    else:
        ops, paths, clr, target = _paint_case(c, rng)
        w, h = c["w"], c["h"]
    # about the time it takes: pieces of edges, and planes of pixels
    segs, n = len(ops), len(paths)
    pieces = segs * (4 if c["pen"] else 1) * 1.5 * (w + h)
    if pieces * 1e-7 + n * w * h * 1e-7 > 20:
        return None
    v, *rest = _strokes_outline(ops, paths) if c["pen"] else _fills(ops, paths)
    cov = _Cover.apply(*rest, n, w, h, c.get("evenodd", False))
    if c["kind"] == "adjoint":
        ((cov - torch.from_numpy(target.astype(np.float64))) ** 2).sum().backward()
        return {"cov": cov.detach().numpy(), "g_ops": v.grad.numpy(), "g_width": None}
    k = torch.from_numpy(clr.astype(np.float64))
    canvas = torch.zeros((w * h, 4), dtype=torch.float64)
    planes = cov.reshape(n, w * h)
    # C = c cov + C (1 - a cov), and back without keeping every canvas
    kept = [canvas]
    with torch.no_grad():
        for i in range(n):
            f = planes[i][:, None]
            canvas = k[i] * f + canvas * (1 - k[i, 3] * f)
            kept.append(canvas if (i + 1) % 20 == 0 else None)
        g = 2 * (canvas - torch.from_numpy(target.astype(np.float64)))
        g_cov = torch.empty((n, w * h), dtype=torch.float64)
        for b in range((n - 1) // 20 * 20, -1, -20):
            run_, part = [kept[b]], min(n, b + 20)
            for i in range(b, part - 1):
                f = planes[i][:, None]
                run_.append(k[i] * f + run_[-1] * (1 - k[i, 3] * f))
            for i in range(part - 1, b - 1, -1):
                g_cov[i] = (g * (k[i] - k[i, 3] * run_[i - b])).sum(1)
                g = g * (1 - k[i, 3] * planes[i][:, None])
    cov.backward(g_cov.reshape(-1))
    return {"out": canvas.numpy(), "g_ops": v.grad.numpy(), "g_width": None}
