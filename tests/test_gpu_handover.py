"""Paths that the tile rasteriser hands over, and uneven ones (dense ops first, or last) that it may
keep: drawn bit-exactly whichever kernel takes them, and in that kernel's time."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300.plotter import fill_batch, pack_batch
from helpers import assert_same, gpu_vs_oracle

pytestmark = pytest.mark.gpu


def uneven(seed, side, big, small, dense_first):
    """`big` long curves and `small` short lines, one after the other."""
    rng = np.random.default_rng(seed)
    curves = workloads.random_path(rng, side, big, n_sub=1)
    lines = workloads.random_path(rng, side, small, n_sub=1)
    lines["kind"] = np.where((lines["kind"] == _abi.OP_QUAD) | (lines["kind"] == _abi.OP_CUBIC), _abi.OP_LINE, lines["kind"])
    return np.concatenate([curves, lines] if dense_first else [lines, curves])


@pytest.mark.parametrize("dense_first", [True, False])
@pytest.mark.parametrize("big,small", [(600, 3000), (130, 4000), (2000, 600)])
def test_uneven_paths(ctx, big, small, dense_first):
    parts = [uneven(k, 200, big, small, dense_first) for k in range(3)]
    for n in (3, 330):  # row ranges, and paths whole
        ops, paths, size = pack_batch([parts[k % 3] for k in range(n)], [200] * n)
        want, got = np.zeros(size, np.uint8), np.zeros(size, np.uint8)
        oracle.fill_batch(0, _abi.NONZERO, ops, paths, 0, want, n_threads=8)
        fill_batch(ctx, ops, paths, 0, got)
        assert_same(got, want, f"{n} paths")
    got, want, *_ = gpu_vs_oracle(ctx, parts[0], 200, 170, rule=_abi.EVENODD, fmt=_abi.RGBA8P, clr=(9, 8, 7, 99), init=37)
    assert_same(got, want, "single call")


def test_handed_over_paths_take_their_kernels_time(ctx):
    """Few large paths, all handed over, against the same batch sent to the CTA rasteriser outright:
    the hand-over may not double the time (1.84 times it with one CTA per SM behind the tile
    rasteriser, 0.97 now)."""
    import torch
    from footile_gb300.plotter import PreparedBatch

    rng = np.random.default_rng(2)
    ops, paths, size = pack_batch([workloads.random_path(rng, 512, 3000)] * 300, [512] * 300)
    dev = torch.from_numpy(ops.view(np.uint8)).cuda()
    ras = torch.zeros(size, dtype=torch.uint8, device="cuda")

    def ms(side):
        ctx.tune(warp_max_side=side)
        batch, took = PreparedBatch(ctx, paths), []
        for _ in range(7):
            batch.launch(dev, ras)
            took.append(ctx.last_ms())
        batch.close()
        return sorted(took)[3]

    by_cta, handed_over = ms(0), ms(512)
    assert handed_over < 1.4 * by_cta, (handed_over, by_cta)


def test_dense_first_path_keeps_the_tile_rasteriser(ctx):
    """1,500 curves, then 6,000 lines: slots for the whole path at the curves' rate would not fit, the
    path does.  The tile rasteriser draws it in a fourth of the CTA rasteriser's time."""
    import torch
    from footile_gb300.plotter import PreparedBatch

    ops, paths, size = pack_batch([uneven(1, 700, 1500, 6000, True)] * 8, [700] * 8)
    dev = torch.from_numpy(ops.view(np.uint8)).cuda()
    ras = torch.zeros(size, dtype=torch.uint8, device="cuda")

    def ms(side):
        ctx.tune(warp_max_side=side)
        batch, took = PreparedBatch(ctx, paths), []
        for _ in range(7):
            batch.launch(dev, ras)
            took.append(ctx.last_ms())
        batch.close()
        return sorted(took)[3]

    by_cta, by_tile = ms(0), ms(512)
    assert by_tile < 0.6 * by_cta, (by_tile, by_cta)
