"""The tile rasteriser's view of a figure (footile_gb300/csrc/ft_tile.cu), restated in numpy
and compared with footile's sequential figure: the same edges whether or not coincident and
closing vertices are dropped, and the same direction from the non-zero segments alone.  And
its Fixed division against exact integers."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi
from footile_gb300.path import PathOp, ops_array


def sequential_figure(ops):
    """Fig::add_point / close (fig.rs:373-461) over Move/Line/Close ops: kept vertices and
    the first vertex of each one's sub-figure."""
    pts, sub = [], []
    start, prev = None, None

    def close():
        nonlocal start
        if start is not None and pts[start:] and prev == first:
            pts.pop(), sub.pop()
        start = None

    first = None
    pending = True
    for o in ops:
        k = int(o["kind"])
        if k in (_abi.OP_MOVE, _abi.OP_CLOSE):
            close()
            pending = True
        if k in (_abi.OP_MOVE, _abi.OP_LINE):
            p = tuple(int(v) for v in np.trunc(o["v"][:2].astype(np.float64) * 65536))
            if pending or start is None:
                start, first, pending = len(pts), p, False
                pts.append(p), sub.append(start)
            elif p != prev:
                pts.append(p), sub.append(start)
            prev = p
    close()
    return pts, sub


def edges_and_direction(pts, sub):
    """Edges with their sense, and the direction of the figure (fig.rs:402-411)."""
    n, edges = len(pts), []
    for i in range(n):
        j = i + 1 if i + 1 < n and sub[i + 1] == sub[i] else sub[i]
        if pts[i][1] != pts[j][1]:
            edges.append((pts[i], pts[j]))
    if not n:
        return sorted(edges), None
    t = min(range(n), key=lambda i: (pts[i][1], pts[i][0], i))
    nf = t + 1 if t + 1 < n and sub[t + 1] == sub[t] else sub[t]
    nr = t - 1 if t > sub[t] else max(i for i in range(n) if sub[i] == sub[t])
    return sorted(edges), turn(pts[nr], pts[t], pts[nf])


def turn(a, p, b):
    m = [int(np.int32(np.uint32(v & 0xFFFFFFFF))) for v in (a[0] - p[0], a[1] - p[1], b[0] - p[0], b[1] - p[1])]
    return 0 if (m[0] * m[3] >> 16) > (m[2] * m[1] >> 16) else 1


def tile_figure(ops):
    """Every op a segment from the pen, every sub-figure closed by one: slots in order, and
    which of them close; then the edges, and the direction from the non-zero segments."""
    segs, closing = [], []
    pen, kind, last, first = (0, 0), None, None, None
    for o in list(ops) + [None]:
        k = None if o is None else int(o["kind"])
        p = None
        if k in (_abi.OP_MOVE, _abi.OP_LINE):
            p = tuple(int(v) for v in np.trunc(o["v"][:2].astype(np.float64) * 65536))
        starts = p is not None and (k == _abi.OP_MOVE or kind in (None, _abi.OP_CLOSE))
        if (starts or o is None) and last is not None:
            closing.append(len(segs))
            segs.append((last, first))
        if p is not None:
            segs.append((p, p) if starts else (pen, p))
            first = p if starts else first
            last = p
        if k in (_abi.OP_MOVE, _abi.OP_LINE, _abi.OP_CLOSE):
            pen, kind = (p if p is not None else (0, 0)), k
    real = [i for i, (a, b) in enumerate(segs) if a != b]
    edges = sorted((a, b) for a, b in segs if a[1] != b[1])
    if not real:
        return edges, None
    t = min(real, key=lambda i: (segs[i][0][1], segs[i][0][0], i))
    lo = max([c + 1 for c in closing if c < t], default=0)
    hi = min(c for c in closing if c >= t)
    before = [i for i in real if lo <= i < t] or [i for i in real if t <= i <= hi]
    return edges, turn(segs[before[-1]][0], segs[t][0], segs[t][1])


@pytest.mark.parametrize("seed", range(60))
def test_edges_and_direction(seed):
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(int(rng.integers(1, 6))):
        # few distinct points: coincident vertices, returns to the start, tied tops
        grid = rng.integers(0, int(rng.integers(2, 6)), (int(rng.integers(1, 14)), 2)).astype(float) / 4 + 1
        if rng.random() < 0.8:
            ops.append(PathOp.Move(*grid[0]))
        ops += [PathOp.Line(*p) for p in grid]
        if rng.random() < 0.3:
            ops.append(PathOp.Line(*grid[0]))
        if rng.random() < 0.6:
            ops.append(PathOp.Close())
    ops = ops_array(ops)
    pts, sub = sequential_figure(ops)
    assert [tuple(int(v) for v in p) for p in oracle.fig_points(ops)] == pts  # the restatement is footile's figure
    assert tile_figure(ops) == edges_and_direction(pts, sub)


def quot(n, d, wobble):
    """fx_quot of ft_tile.cu in numpy: `wobble` moves the approximate reciprocal by an ulp
    either way (rcp.approx is within one)."""
    f32, u32 = np.float32, np.uint32
    f = (f32(1) / d.astype(f32)).astype(f32)
    f = np.nextafter(f, np.where(wobble > 0, f32(np.inf), f32(0)), dtype=f32) if wobble else f
    est = n.astype(f32) * f * f32(65536)
    q = est.astype(np.uint64).astype(u32)
    r = ((n << u32(16)) - q * d).astype(np.int32)
    q2 = np.rint(r.astype(f32) * f).astype(np.int32)
    r = (r.astype(u32) - q2.astype(u32) * d).astype(np.int32)
    return q + q2.astype(u32) - (r < 0).astype(u32) + (r >= d.astype(np.int32)).astype(u32), est < f32(2147483000.0)


@pytest.mark.parametrize("wobble", [-1, 0, 1])
def test_division(wobble):
    rng = np.random.default_rng(7)
    n = np.exp2(rng.uniform(0, 28, 2_000_000)).astype(np.uint32)
    d = np.exp2(rng.uniform(0, 28, 2_000_000)).astype(np.uint32)
    edge = np.array([1, 2, 3, 65535, 65536, 65537, 2**21, 2**24 - 1, 2**24 + 1, 2**28 - 1], np.uint32)
    k = rng.integers(1, 2**16, 200_000).astype(np.uint32)
    m = rng.integers(1, 2**12, 200_000).astype(np.uint32)
    # exact multiples and their neighbours, where a unit is lost first
    n = np.concatenate([n, np.repeat(edge, len(edge)), k * m, k * m + 1, k * m - 1])
    d = np.concatenate([d, np.tile(edge, len(edge)), m, m, m])
    n, d = np.minimum(n, 2**28 - 1), np.maximum(d, 1)
    got, taken = quot(n, d, wobble)
    want = (n.astype(np.uint64) << np.uint64(16)) // d.astype(np.uint64)
    assert np.array_equal(got[taken], want[taken].astype(np.uint32))
    assert (want[~taken] > 2**31 - 2**12).all()
