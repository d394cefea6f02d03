"""Coverage gradients beside an edge: a cell that an edge only touches on its left border holds
none of the edge, so whatever gradient stands there (inf and NaN too) must not reach the edge's
vertices."""
import numpy as np
import pytest

from footile_gb300 import _abi
from footile_gb300.adjoint import Adjoint
from footile_gb300.path import PathOp, ops_array
from footile_gb300.plotter import pack_batch

pytestmark = pytest.mark.gpu
M, L, Z = PathOp.Move, PathOp.Line, PathOp.Close

# (points, cells touched from the left only): edges that end, within a row, on a column's border;
# an edge leaving the raster's left side at x = 0; a long flat edge over many cells
SHAPES = [
    ([(1, 1), (4, 2), (1, 3)], [(1, 4), (2, 4)]),
    ([(6, 1), (2, 1.5), (2, 2.5), (6, 3), (3, 2)], [(1, 6), (2, 6)]),
    ([(-3, 2), (0, 2.75), (-3, 3.25)], [(2, 0), (3, 0)]),
    ([(0.5, 4.25), (13, 4.5), (0.5, 4.75)], [(4, 13)]),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("rule", [_abi.NONZERO, _abi.EVENODD])
def test_cells_touched_from_the_left_are_not_read(ctx, shape, bad, rule):
    pts, cells = shape
    side = 16
    path = ops_array([M(*pts[0])] + [L(*p) for p in pts[1:]] + [Z()])
    ops, paths, _ = pack_batch([path], [side])
    paths["stride"] = 4 * side
    adj = Adjoint(ctx)
    try:
        adj.forward(rule, ops, paths, np.zeros((side, side), np.float32))
        g = np.random.default_rng(3).random((side, side)).astype(np.float32)
        for r, c in cells:
            g[r, c] = 0
        want = adj.backward(g, np.zeros((len(ops), 6), np.float32))
        for r, c in cells:
            g[r, c] = bad
        got = adj.backward(g, np.zeros((len(ops), 6), np.float32))
    finally:
        adj.close()
    assert np.isfinite(got).all()
    # the same sums, of atomics in an order of their own: a few roundings of the largest
    assert np.abs(got - want).max() <= 8 * np.finfo(np.float32).eps * np.abs(want).max()
