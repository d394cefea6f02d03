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
