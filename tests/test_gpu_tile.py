"""The tile rasteriser against the oracle, bit-exact, where it can go wrong: canvas sizes
around its lanes, bands and row routes; figures with negative top rows, degenerate and
re-opened sub-figures, tied tops; slopes at both ends of the Fixed range; paths it hands to
the CTA rasteriser."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.path import PathOp, ops_array
from footile_gb300.plotter import fill_batch, pack_batch
from helpers import assert_same, gpu_vs_oracle

pytestmark = pytest.mark.gpu


def batch_vs_oracle(ctx, per_path, sizes, fmt, rule, host=False, pad=0, tolerance=0.3):
    """One batch of more than two paths per SM (whole canvases, 128 threads each)."""
    torch = pytest.importorskip("torch")
    n = 320
    rng = np.random.default_rng(5)
    per_path, sizes = [per_path[i % len(per_path)] for i in range(n)], [sizes[i % len(sizes)] for i in range(n)]
    clrs = rng.integers(0, 256, (n, 4)).astype(np.uint8)
    ops, paths, nbytes = pack_batch(per_path, sizes, fmt, clrs)
    if pad >= 0 and fmt == _abi.MATTE8:  # rows of `pad` spare bytes, rasters at any byte
        paths["stride"] = paths["width"] + pad
        size = paths["stride"].astype(np.int64) * paths["height"] + pad
        paths["raster_offset"] = np.cumsum(size) - size
        nbytes = int(size.sum())
    init = rng.integers(0, 256, nbytes).astype(np.uint8)
    want = init.copy()
    st_o = oracle.fill_batch(0, rule, ops, paths, fmt, want, n_threads=8, tolerance=tolerance)
    ctx.set_tolerance(tolerance)
    if host:
        pin = torch.from_numpy(init.copy()).pin_memory()
        st = fill_batch(ctx, ops, paths, fmt, pin.numpy(), rule)
        got = pin.numpy()
    else:
        ras = torch.from_numpy(init.copy()).cuda()
        st = fill_batch(ctx, torch.from_numpy(ops.view(np.uint8)).cuda(), paths, fmt, ras, rule)
        got = ras.cpu().numpy()
    assert np.array_equal(st, st_o)
    assert_same(got, want, "batch")


SIDES = [1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300, 511, 512]


def random_paths(seed, sizes, spread=1.0):
    rng = np.random.default_rng(seed)
    out = []
    for w, h in sizes:
        ops = workloads.random_path(rng, 1.0, int(rng.integers(3, 40)), n_sub=int(rng.integers(1, 4)))
        ops["v"][:, 0::2] = (ops["v"][:, 0::2] - 0.5) * w * spread + 0.5 * w
        ops["v"][:, 1::2] = (ops["v"][:, 1::2] - 0.5) * h * spread + 0.5 * h
        out.append(ops)
    return out


@pytest.mark.parametrize("rule", [_abi.NONZERO, _abi.EVENODD])
@pytest.mark.parametrize("fmt,host,pad", [(_abi.MATTE8, False, -1), (_abi.MATTE8, False, 1), (_abi.MATTE8, True, 0),
                                          (_abi.MATTE8, True, 3), (_abi.RGBA8P, False, -1)])
def test_sizes(ctx, rule, fmt, host, pad):
    rng = np.random.default_rng(11)
    sizes = [(w, int(rng.choice(SIDES))) for w in SIDES] + [(int(rng.choice(SIDES)), h) for h in SIDES]
    # figures inside the canvas, and reaching over every side of it
    per_path = random_paths(1, sizes) + random_paths(2, sizes, 3.0)
    batch_vs_oracle(ctx, per_path, sizes + sizes, fmt, rule, host, pad)


def odd_figures():
    M, L, Q, C, Z, W = PathOp.Move, PathOp.Line, PathOp.Quad, PathOp.Cubic, PathOp.Close, PathOp.PenWidth
    nan = float("nan")
    square = [M(4, 4), L(20, 4), L(20, 20), L(4, 20)]
    yield "nothing", [Z()]
    yield "moves", [M(3, 3), M(5, 5), M(3, 1)]
    yield "degenerate sub-figure on top", [M(9, 1), L(9, 1), Z()] + square
    yield "coincident vertices", [M(4, 4), L(4, 4), L(20, 4), L(20, 4), L(20, 20), L(4, 20), L(4, 4), L(4, 4), Z()]
    yield "line after a close", square + [Z(), L(30, 3), L(25, 25), L(40, 20)]
    yield "quad after a close", square + [Z(), Q(50, 0, 30, 40), L(3, 30)]
    yield "cubic first", [C(60, 0, 0, 60, 40, 40), L(3, 30)]
    yield "tied tops, reversed second", square + [Z(), M(4, 4), L(4, 30), L(30, 30), L(30, 4)]
    yield "reversed", [M(4, 20), L(20, 20), L(20, 4), L(4, 4), Z()]
    yield "above the canvas", [M(-5, -300.5), L(50, -20.25), L(30, 70), L(-40, 33)]
    yield "near horizontal", [M(0, 10), L(63, 10.00002), L(63, 30.5), L(0, 30.49998)]
    yield "near vertical", [M(10.00002, 0), L(10, 63), L(40, 63), L(40.00002, 0)]
    yield "steep beyond 32,768", [M(10, -32000), L(10.0001, 32000), L(30, 32000), L(30, -32000)]
    yield "flat beyond the canvas", [M(-30000, 10.25), L(30000, 11), L(30000, 40), L(-30000, 39.5)]
    yield "off the Fixed range", [M(-1e6, -1e6), L(1e6, 5), L(30, 1e6)]
    yield "not a number", square + [Q(nan, 3, 9, 9), L(5, 40)]
    yield "infinite", square + [C(3, 3, float("inf"), 3, 9, 9), L(5, 40)]
    yield "pen widths between", [W(3), M(4, 4), W(2), L(20, 4), W(5), Q(40, 10, 20, 20), Z(), W(7)]
    yield "flat loops", [M(5, 5), C(60, 5, 5, 60, 60, 60), C(5, 60, 60, 5, 5, 5), Z()]
    yield "collinear cubic", [M(5, 5), C(20, 20, 40, 40, 60, 60), L(5, 60)]
    yield "one segment cubic S", [M(5, 5), C(5, 60, 60, 5, 60, 60), Z()]
    yield "ops over a chunk", [M(1, 1)] + [L(1 + (i * 37) % 61, 1 + (i * 23) % 59) for i in range(700)]
    yield "closes at a chunk's edge", sum(([M(i % 50, 3), L(60, i % 60), L(2, 60), Z()] for i in range(160)), [])


@pytest.mark.parametrize("name,ops", list(odd_figures()), ids=lambda v: v if isinstance(v, str) else "")
def test_odd_figures(ctx, name, ops):
    ops = ops_array(ops)
    for fmt in (_abi.MATTE8, _abi.RGBA8P):
        got, want, st, sw, err = gpu_vs_oracle(ctx, ops, 64, 67, fmt, _abi.NONZERO, (9, 200, 31, 210), 77)
        assert_same(got, want, f"{name}, few")
        assert (err is None) == (st == 0) and ctx.pen_width() == sw
    batch_vs_oracle(ctx, [ops], [(64, 67)], _abi.MATTE8, _abi.EVENODD, pad=-1)


@pytest.mark.parametrize("tolerance,scale", [(0.01, 1.0), (0.01, 300.0), (0.3, 20000.0)])
def test_handed_over(ctx, tolerance, scale):
    """Curves deeper than a slot walks, more slots than the scratch holds: drawn by the CTA
    rasteriser, mixed with paths that stay."""
    rng = np.random.default_rng(3)
    big = workloads.random_path(rng, 100.0 * scale, 60)
    many = workloads.random_path(rng, 256, 400, probs=(0, 0, 1), n_sub=4)  # 1,600 long cubics
    small = workloads.random_path(rng, 100, 12)
    batch_vs_oracle(ctx, [big, small, many], [(100, 90), (100, 100), (256, 256)], _abi.MATTE8, _abi.NONZERO, pad=-1,
                    tolerance=tolerance)
    for ops in (big, many):
        got, want, _, _, _ = gpu_vs_oracle(ctx, ops, 120, 100, _abi.RGBA8P, clr=(50, 60, 70, 128), tolerance=tolerance)
        assert_same(got, want, "few")


@pytest.mark.parametrize("w,h", [(256, 256), (1, 3000), (3000, 1), (900, 700), (1021, 1009), (517, 40)])
def test_few_paths(ctx, w, h):
    for ops, fmt in zip(random_paths(w, [(w, h)] * 2, 1.2), (_abi.MATTE8, _abi.RGBA8P)):
        got, want, _, _, _ = gpu_vs_oracle(ctx, ops, w, h, fmt, clr=(50, 60, 70, 128), init=33)
        assert_same(got, want, f"{w}x{h}")
