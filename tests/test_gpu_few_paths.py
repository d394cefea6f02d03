"""Batches of few paths on large canvases (row ranges of the tile rasteriser, with one and with two
CTAs per SM): the oracle's bytes, and no more time than the CTA rasteriser takes for them."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.plotter import PreparedBatch, fill_batch, pack_batch
from helpers import assert_same

pytestmark = pytest.mark.gpu


def batch(n, w, h, fmt, seed=4):
    rng = np.random.default_rng(seed)
    return pack_batch([workloads.random_path(rng, min(w, h), 6) for _ in range(n)], [(w, h)] * n, fmt,
                      rng.integers(0, 256, (n, 4)))


@pytest.mark.parametrize("n,w,h", [(1, 900, 900), (2, 17, 30000), (40, 130, 900), (152, 310, 40), (153, 310, 40),
                                   (290, 301, 170), (300, 1000, 33)])
@pytest.mark.parametrize("fmt", [_abi.MATTE8, _abi.RGBA8P])
def test_row_ranges(ctx, n, w, h, fmt):
    ops, paths, size = batch(n, w, h, fmt)
    want = np.random.default_rng(1).integers(0, 256, size).astype(np.uint8)
    got = want.copy()
    oracle.fill_batch(0, _abi.NONZERO, ops, paths, fmt, want, n_threads=8)
    fill_batch(ctx, ops, paths, fmt, got)
    assert_same(got, want, f"{n} x {w}x{h}")


@pytest.mark.parametrize("w", [257, 260, 511, 512, 900])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_wide_mask_rows(ctx, w, pad):
    """Rows wider than a warp's 256 pixels on any boundary, whole in a batch and by ranges."""
    for n in (3, 320):
        ops, paths, _ = batch(n, w, 21, _abi.MATTE8, w)
        paths["stride"] = w + pad
        size = (w + pad) * 21
        paths["raster_offset"] = np.arange(n) * size
        want = np.random.default_rng(1).integers(0, 256, n * size).astype(np.uint8)
        got = want.copy()
        oracle.fill_batch(0, _abi.EVENODD, ops, paths, _abi.MATTE8, want, n_threads=8)
        fill_batch(ctx, ops, paths, _abi.MATTE8, got, _abi.EVENODD)
        assert_same(got, want, f"{n} x {w}+{pad}")


@pytest.mark.parametrize("n", [40, 120, 300])
def test_no_slower_than_the_cta_rasteriser(ctx, n):
    """(1.6, 1.9 and 2.0 times its time with one CTA per SM and one load in flight per lane.)"""
    import torch

    ops, paths, size = batch(n, 900, 900, _abi.RGBA8P)
    dev = torch.from_numpy(ops.view(np.uint8)).cuda()
    ras = torch.zeros(size, dtype=torch.uint8, device="cuda")

    def ms(side):
        ctx.tune(warp_max_side=side)
        b, took = PreparedBatch(ctx, paths, _abi.RGBA8P), []
        for _ in range(9):
            b.launch(dev, ras)
            took.append(ctx.last_ms())
        b.close()
        return sorted(took)[4]

    by_cta, tiled = ms(0), ms(512)
    assert tiled < 1.3 * by_cta, (tiled, by_cta)


@pytest.mark.parametrize("w,h", [(128, 128), (149, 134), (149, 135), (117, 133), (117, 134)])
@pytest.mark.parametrize("fmt", [_abi.MATTE8, _abi.RGBA8P])
def test_bands_of_two_ctas(ctx, w, h, fmt):
    """A path in one band of its cells, in two: on both sides of what two CTAs per SM leave room for,
    20,400 cells, 16,000 where rows are staged."""
    test_row_ranges(ctx, 200, w, h, fmt)
