"""The ordered Rgba8p compositor against the oracle, bit-exact, where its tiles can go wrong:
rows of one to four segments and of more (edges binned by segment, sums handed from warp to
warp, or every edge walked by every segment), canvases staged or in place, calls cut into
batches, figures that cover whole segments or reach far over the canvas."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.path import PathOp, ops_array
from footile_gb300.plotter import composite_batch, pack_batch
from helpers import assert_same

pytestmark = pytest.mark.gpu


def calls(seed, n, w, h, stroke):
    """Curves over and beyond the canvas, rectangles over most of it, far and flat triangles."""
    rng = np.random.default_rng(seed)
    out, clrs = [], []
    M, L, Z = PathOp.Move, PathOp.Line, PathOp.Close
    for i in range(n):
        if i % 4 == 1:
            x0, x1 = np.sort(rng.uniform(-0.2, 1.2, 2)) * w
            y0, y1 = np.sort(rng.uniform(-0.2, 1.2, 2)) * h
            o = ops_array([M(x0, y0), L(x1, y0 + 0.3), L(x1, y1), L(x0, y1), Z()])
        elif i % 8 == 2:
            far = float(rng.choice([9000, 40000, 1e6]))
            o = ops_array([M(-far, rng.uniform(0, h)), L(far, rng.uniform(0, h)), L(rng.uniform(0, w), far), Z()])
        else:
            o = workloads.random_path(rng, 1.0, int(rng.integers(2, 24)), close=not stroke or i % 3 == 0)
            o["v"][:, 0::2] = (o["v"][:, 0::2] * 1.6 - 0.3) * w
            o["v"][:, 1::2] = (o["v"][:, 1::2] * 1.6 - 0.3) * h
        if stroke:
            o = np.concatenate([ops_array([PathOp.PenWidth(float(rng.uniform(1, 30)))]), o])
        a = int(rng.integers(30, 256))
        out.append(o)
        clrs.append([int(v) * a // 255 for v in rng.integers(0, 40 if i % 2 else 256, 3)] + [a])
    ops, paths, _ = pack_batch(out, [(w, h)] * n, _abi.RGBA8P, clrs)
    return ops, paths, rng.integers(0, 256, (h, w, 4)).astype(np.uint8)


def check(ctx, n, w, h, stroke, rule, seed=1):
    ops, paths, init = calls(seed, n, w, h, stroke)
    want, got = init.copy(), init.copy()
    st_o, _ = oracle.composite(int(stroke), rule, ops, paths, _abi.RGBA8P, want, s_width=1.0)
    ctx.set_pen_width(1.0)
    st = composite_batch(ctx, ops, paths, _abi.RGBA8P, got, rule, stroke=stroke)
    assert (st == st_o).all()
    assert_same(got, want, f"{w}x{h}")


@pytest.mark.parametrize("w,tile_w,band_rows", [
    (1, 0, 0), (127, 0, 0), (128, 0, 0), (129, 0, 0), (255, 0, 5), (300, 0, 0), (513, 0, 0), (800, 0, 8), (1100, 0, 0),
    (1300, 512, 3), (500, 128, 2), (512, 128, 6), (640, 128, 0), (2048, 512, 1), (2049, 1024, 4), (4097, 1024, 0),
    (4300, 0, 0), (257, 1024, 7)])
@pytest.mark.parametrize("staged", [True, False])
def test_segments(ctx, w, tile_w, band_rows, staged):
    ctx.tune(tile_w=tile_w, band_rows=band_rows, tile_stage=1 if staged else 2)
    try:
        check(ctx, 40, w, 61, True, _abi.NONZERO)
        check(ctx, 40, w, 67, False, _abi.EVENODD if w % 2 else _abi.NONZERO, 2)
    finally:
        ctx.set_tuning(None)


@pytest.mark.parametrize("n", [63, 64, 130])
def test_batches_of_calls(ctx, n):
    """More tiles than the GPU holds at once: 64 calls are two batches, the last of 130 short."""
    check(ctx, n, 1060, 3701, False, _abi.NONZERO, n)


def test_many_calls_on_few_rows(ctx):
    """Rounds of 32 calls with the ring of sums between segments full, and calls that do not
    reach the rows."""
    check(ctx, 700, 700, 19, True, _abi.NONZERO)
