"""Device memory goes back with the context that took it."""
import numpy as np
import pytest

from footile_gb300 import _abi, workloads
from footile_gb300._lib import Context
from footile_gb300.path import FillRule, PathOp, ops_array
from footile_gb300.plotter import Plotter, composite_batch, fill_batch, pack_batch

pytestmark = pytest.mark.gpu


def draw_everything():
    """Small, large and batched calls, so that every buffer of a context is taken."""
    ctx = Context(0)
    rng = np.random.default_rng(5)
    big = workloads.random_path(rng, 1200, 3000)
    for stroke in (False, True):  # built over the whole GPU, Matte8 and through the mask
        for shape in ((1100, 1200), (1100, 1200, 4), (60, 70)):
            p = Plotter(np.zeros(shape, np.uint8), context=ctx)
            ops = np.concatenate([ops_array([PathOp.PenWidth(3.0)]), big]) if stroke else big
            p.stroke(ops, (1, 2, 3, 255)) if stroke else p.fill(FillRule.NonZero, ops, (1, 2, 3, 255))
    ops, paths, nbytes = pack_batch([workloads.random_path(rng, 64, 10) for _ in range(400)], [64] * 400)
    fill_batch(ctx, ops, paths, 0, np.zeros(nbytes, np.uint8))
    composite_batch(ctx, ops, paths, _abi.RGBA8P, np.zeros((300, 300, 4), np.uint8))
    raster = np.zeros((64, 64, 4), np.uint8)
    ctx.convert(raster, raster.copy())
    ctx.close()


def test_a_closed_context_gives_its_memory_back(cuda_ok, gpu_lib):
    import torch

    draw_everything()  # the library's kernels load
    free = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        draw_everything()
    # the buffers of one context take hundreds of megabytes; allocations come in 2 MB pieces
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20


def test_a_composite_needs_no_bins_by_segment(cuda_ok, gpu_lib):
    """100,000 calls on 512 x 12,000 pixels: their bins' offsets take 1.2 GB by band, 4.8 GB by
    segment as well, beside 4.4 GB of build scratch.  With 6.6 GB free the call is drawn as with
    all of the memory."""
    import torch

    n, w, h = 100_000, 512, 12_000
    rng = np.random.default_rng(9)
    ops = np.zeros((n, 4), _abi.OP_DTYPE)
    ops["kind"] = [_abi.OP_MOVE, _abi.OP_LINE, _abi.OP_LINE, _abi.OP_CLOSE]
    at = rng.random((n, 1, 2)) * [w, h] + rng.random((n, 3, 2)) * 40 - 20
    ops["v"][:, :3, :2] = at
    paths = np.zeros(n, _abi.PATH_DTYPE)
    paths["op_begin"], paths["n_ops"] = np.arange(n) * 4, 4
    paths["clr"] = rng.integers(0, 256, (n, 4))
    paths["clr"][:, :3] = np.minimum(paths["clr"][:, :3], paths["clr"][:, 3:])
    dev = torch.from_numpy(ops.reshape(-1).view(np.uint8)).cuda()

    def draw():
        ctx = Context(0)
        try:
            ctx.tune(tile_w=128, pool_edges=1 << 21)
            raster = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
            assert (composite_batch(ctx, dev, paths, _abi.RGBA8P, raster) == _abi.OK).all()
            ctx.sync()
            return raster.cpu().numpy()
        finally:
            ctx.close()

    want = draw()
    torch.cuda.empty_cache()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - int(6.6e9), dtype=torch.uint8, device="cuda")
    try:
        got = draw()
    finally:
        del taken
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)
