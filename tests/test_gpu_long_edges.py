"""Ordered composites of figures with edges over hundreds of bands (closing lines, rectangles, far
triangles) beside short ones: binned over a warp's lanes, the oracle's bytes."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.path import PathOp, ops_array
from footile_gb300.plotter import composite_batch, pack_batch
from helpers import assert_same

pytestmark = pytest.mark.gpu
M, L, Z = PathOp.Move, PathOp.Line, PathOp.Close


@pytest.mark.parametrize("w,h,band_rows", [(300, 132, 1), (300, 133, 1), (700, 1100, 0), (130, 2100, 8), (1100, 400, 2)])
@pytest.mark.parametrize("fmt", [_abi.RGBA8P, _abi.MATTE8])
@pytest.mark.parametrize("stroke", [False, True])
def test_long_edges(ctx, w, h, band_rows, fmt, stroke):
    rng = np.random.default_rng(w + h)
    parts = []
    for k in range(24):
        n = [3, 40, 300][k % 3]  # edges of one warp, of several, of more than a step
        x, y = rng.uniform(-0.1, 1.1, n) * w, rng.uniform(-0.2, 1.2, n) * h
        y[rng.random(n) < 0.5] = rng.uniform(0, h)  # short ones among them
        parts.append(ops_array([M(x[0], y[0])] + [L(a, b) for a, b in zip(x[1:], y[1:])] + [Z()]))
        parts.append(workloads.random_path(rng, min(w, h), 12))
    ops, paths, _ = pack_batch(parts, [(w, h)] * len(parts), fmt, rng.integers(0, 120, (len(parts), 4)) + [0, 0, 0, 130])
    init = rng.integers(0, 256, (h, w, 4) if fmt == _abi.RGBA8P else (h, w)).astype(np.uint8)
    want, got = init.copy(), init.copy()
    oracle.composite(int(stroke), _abi.NONZERO, ops, paths, fmt, want, s_width=1.0)
    ctx.set_pen_width(1.0)
    ctx.tune(band_rows=band_rows)
    try:
        composite_batch(ctx, ops, paths, fmt, got, stroke=stroke)
    finally:
        ctx.set_tuning(None)
    assert_same(got, want, f"{w}x{h}")
