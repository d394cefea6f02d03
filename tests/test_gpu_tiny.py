"""Batches of tiny canvases (the tile rasteriser by one warp a path) against the oracle, bit-exact, at
the edges of what counts as tiny, and with paths beside them that are not."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.path import PathOp, ops_array
from footile_gb300.plotter import fill_batch, pack_batch
from helpers import assert_same

pytestmark = pytest.mark.gpu


def run(ctx, parts, sizes, fmt, rule, pad=0, host=False):
    ops, paths, size = pack_batch(parts, sizes, fmt, np.random.default_rng(2).integers(0, 256, (len(parts), 4)))
    bpp = _abi.BYTES_PER_PIXEL[fmt]
    paths["stride"] = paths["width"] * bpp + pad * bpp
    rows = paths["stride"].astype(np.int64) * paths["height"]
    paths["raster_offset"], size = np.cumsum(rows) - rows, int(rows.sum())
    want = np.random.default_rng(1).integers(0, 256, size).astype(np.uint8)
    if host:
        import torch
        keep = torch.from_numpy(want.copy()).pin_memory()
        got = keep.numpy()
    else:
        got = want.copy()
    st_o = oracle.fill_batch(0, rule, ops, paths, fmt, want, n_threads=8)
    st = fill_batch(ctx, ops, paths, fmt, got, rule)
    assert_same(got, want, f"{fmt} {rule} {pad} {host}")
    return st, st_o


@pytest.mark.parametrize("fmt,rule,pad,host", [(0, 0, 0, False), (0, 1, 1, False), (1, 0, 0, False), (1, 1, 3, False),
                                               (0, 0, 0, True), (0, 1, 5, True)])
@pytest.mark.parametrize("top,n_ops", [(8, 5), (24, 62), (25, 62), (24, 63), (24, 64)])
def test_sides_and_ops(ctx, fmt, rule, pad, host, top, n_ops):
    fmt = _abi.RGBA8P if fmt else _abi.MATTE8
    rng = np.random.default_rng(top + n_ops)
    sizes = [(int(rng.integers(0, top + 1)), int(rng.integers(0, top + 1))) for _ in range(398)] + [(top, top)] * 2
    parts = [workloads.random_path(rng, max(*s, 1), int(rng.integers(1, n_ops + 1))) for s in sizes[:-2]]
    parts += [workloads.random_path(rng, top, n_ops)] * 2  # with its Move and Close: at the limit and above it
    run(ctx, parts, sizes, fmt, rule, pad, host)


def test_far_larger_drawings_and_bad_ops(ctx):
    """Drawings a hundred times the canvas (more slots than a tiny path's scratch: handed over), curves
    too deep for slots, and ops with nothing to draw."""
    rng = np.random.default_rng(9)
    parts = []
    for k in range(400):
        o = workloads.random_path(rng, 20.0, int(rng.integers(2, 50)))
        if k % 4 == 0:
            o["v"] = (o["v"] - 10) * 100
        elif k % 16 == 1:
            o["v"] = (o["v"] - 10) * 4000
        elif k % 16 == 2:
            o["v"][rng.integers(1, len(o)), 0] = np.nan
        elif k % 16 == 3:
            o = ops_array([PathOp.Close(), PathOp.PenWidth(3.0), PathOp.Move(1, 2)])
        parts.append(o)
    run(ctx, parts, [(20, 17)] * 400, _abi.MATTE8, _abi.EVENODD)


def test_one_large_path_among_tiny_ones(ctx):
    rng = np.random.default_rng(4)
    sides = [12] * 399 + [200]
    run(ctx, [workloads.random_path(rng, s, 9) for s in sides], sides, _abi.MATTE8, _abi.NONZERO)


@pytest.mark.parametrize("fmt,rule,pad", [(0, 0, 0), (0, 1, 1), (1, 0, 0), (1, 1, 3)])
@pytest.mark.parametrize("top,n_ops,less", [(8, 3, 0), (24, 16, 0), (24, 17, 0), (25, 16, 0), (24, 16, 1)])
def test_as_many_as_one_warp_a_path_takes(ctx, fmt, rule, pad, top, n_ops, less):
    """128 canvases per SM, and one less; sides and ops at their limits and above."""
    import torch

    n = 128 * torch.cuda.get_device_properties(0).multi_processor_count - less
    rng = np.random.default_rng(top + n_ops)
    some = [workloads.random_path(rng, top, int(rng.integers(1, n_ops - 1))) for _ in range(200)]
    for k in range(0, 200, 5):  # zoomed in: up to the scratch's last slot, and curves too deep for slots
        some[k]["v"] = (some[k]["v"] - top / 2) * (100 if k % 10 else 4000)
    some[1] = workloads.random_path(rng, top, n_ops - 2)
    assert len(some[1]) == n_ops
    sides = rng.integers(1, top + 1, (n, 2))
    sides[1] = top
    run(ctx, [some[k % 200] for k in range(n)], [tuple(int(v) for v in s) for s in sides],
        _abi.RGBA8P if fmt else _abi.MATTE8, rule, pad)


def test_zoomed_in_batches_keep_four_warps(ctx):
    """Curves far larger than 3,000 tiny canvases: a path's chain sets the time, by one warp a path five
    times that of four."""
    import torch
    from footile_gb300.plotter import PreparedBatch

    rng = np.random.default_rng(4)
    parts = [workloads.random_path(rng, 16000, 62, probs=(0, .5, .5)) for _ in range(64)]
    took = []
    for side in (24, 25):  # 25: not tiny
        ops, paths, size = pack_batch([parts[k % 64] for k in range(3000)], [side] * 3000)
        dev = torch.from_numpy(ops.view(np.uint8)).cuda()
        ras = torch.zeros(size, dtype=torch.uint8, device="cuda")
        batch, ms = PreparedBatch(ctx, paths), []
        for _ in range(7):
            batch.launch(dev, ras)
            ms.append(ctx.last_ms())
        batch.close()
        took.append(sorted(ms)[3])
    assert took[0] < 2 * took[1], took
