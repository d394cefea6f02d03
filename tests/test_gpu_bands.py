"""Single calls through the band compositor and the mask passes against the oracle, bit-exact:
band heights, widths that take 1,024, 512 and 256 threads, rows of every alignment, colours that
are opaque and not; and curves too deep for slots in strokes and in the coverage adjoint."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.adjoint import Adjoint, pack_coverage
from footile_gb300.path import PathOp, ops_array
from helpers import assert_same, gpu_vs_oracle

pytestmark = pytest.mark.gpu


def drawing(seed, w, h):
    rng = np.random.default_rng(seed)
    o = workloads.random_path(rng, 1.0, 60, n_sub=5)
    o["v"][:, 0::2] = (o["v"][:, 0::2] * 1.4 - 0.2) * w
    o["v"][:, 1::2] = (o["v"][:, 1::2] * 1.4 - 0.2) * h
    return o


@pytest.mark.parametrize("w,h", [(1, 1), (3, 70), (8, 8), (127, 33), (256, 9), (1021, 40), (1532, 19), (4096, 23),
                                 (6001, 11), (9000, 13), (16383, 10), (16384, 9)])
@pytest.mark.parametrize("band_rows", [0, 1, 3])
def test_bands(ctx, w, h, band_rows):
    ctx.tune(split_px=1, band_rows=band_rows)
    try:
        for k, (fmt, rule, clr) in enumerate([(_abi.MATTE8, _abi.NONZERO, (0, 0, 0, 0)),
                                              (_abi.MATTE8, _abi.EVENODD, (0, 0, 0, 0)),
                                              (_abi.RGBA8P, _abi.NONZERO, (9, 200, 31, 255)),
                                              (_abi.RGBA8P, _abi.EVENODD, (50, 60, 7, 128))]):
            rng = np.random.default_rng(k)
            shape = (h, w) if fmt == _abi.MATTE8 else (h, w, 4)
            init = rng.integers(0, 256 if k % 2 else 24, shape).astype(np.uint8)
            got, want, *_ = gpu_vs_oracle(ctx, drawing(k, w, h), w, h, fmt, rule, clr, init)
            assert_same(got, want, f"{w}x{h} {fmt} {rule}")
    finally:
        ctx.set_tuning(None)


@pytest.mark.parametrize("join", [_abi.JOIN_MITER, _abi.JOIN_BEVEL, _abi.JOIN_ROUND])
def test_deep_curves_in_a_stroke(ctx, join):
    """A curve whose points of 2e4 are not known to be flat at depth 12 at a tolerance of 0.01
    (walked depth first), between ordinary ones."""
    M, Q, C, W = PathOp.Move, PathOp.Quad, PathOp.Cubic, PathOp.PenWidth
    ops = ops_array([W(3), M(5, 5), Q(60, 10, 20, 50), W(6), C(2e4, -1.5e4, -1.8e4, 2e4, 40, 30), Q(10, 60, 55, 5)])
    for split_px in (0, 1):
        ctx.tune(split_px=split_px or 1 << 20)
        try:
            got, want, st, sw, err = gpu_vs_oracle(ctx, ops, 64, 61, stroke=True, join=join, tolerance=0.01)
        finally:
            ctx.set_tuning(None)
        assert_same(got, want, f"join {join}")
        assert (err is None) == (st == 0) and ctx.pen_width() == sw


def test_deep_curves_in_the_adjoint(ctx):
    """Points of 2e4 at a tolerance of 0.01 are not known to be flat at depth 12: the op is walked
    depth first.  One ulp there is 2^-9 px, and a cell's area is a product of differences of such
    numbers, each rounded once: four ulps bound it."""
    M, Q, C, Z = PathOp.Move, PathOp.Quad, PathOp.Cubic, PathOp.Close
    path = ops_array([M(3, 4), Q(30, 2, 28, 20), C(2e4, 25, -2e4, 30, 12, 29), Q(2, 20, 3, 4), Z()])
    ops, paths, nbytes = pack_coverage([path], [(32, 33)])
    ctx.set_tolerance(0.01)
    adj = Adjoint(ctx)
    cov = np.zeros(nbytes // 4, np.float32)
    adj.forward(_abi.NONZERO, ops, paths, cov)
    g = np.zeros((len(ops), 6), np.float32)
    adj.backward(np.ones_like(cov), g)
    assert (adj.status() == 0).all() and np.isfinite(g).all() and g.any()
    adj.close()
    ctx.set_tolerance(0.3)
    want, _, st = oracle.adj_forward(_abi.NONZERO, path, 32, 33, tolerance=0.01)
    assert st == 0
    assert np.abs(cov - want.ravel()).max() < 4 * 2.0 ** -9
