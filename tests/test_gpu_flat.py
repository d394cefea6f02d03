"""Segments far longer than the canvas is wide, against the oracle, bit-exact: their rows go to as
many lanes as the raster has cells for, counted from where the walk enters it."""
import numpy as np
import pytest

import oracle
from footile_gb300 import _abi
from footile_gb300.path import PathOp, ops_array
from footile_gb300.plotter import fill_batch, pack_batch
from helpers import assert_same, gpu_vs_oracle

pytestmark = pytest.mark.gpu


def flat(rng, w, h, half):
    """A closed path of nearly flat segments from far left to far right and back, some that start
    or end on the canvas."""
    x = rng.uniform(-half, half, 24)
    on = rng.random(24) < 0.3
    x[on] = rng.uniform(-2, w + 2, on.sum())
    y = np.clip(np.cumsum(rng.normal(0, 0.6, 24)) + rng.uniform(0, h), -3, h + 3)
    return ops_array([PathOp.Move(x[0], y[0])] + [PathOp.Line(a, b) for a, b in zip(x[1:], y[1:])] + [PathOp.Close()])


@pytest.mark.parametrize("w", [1, 3, 4, 5, 8, 9, 31, 33, 64, 255, 257, 512])
@pytest.mark.parametrize("half", [40, 3000, 16000])
def test_flat_segments_batch(ctx, w, half):
    rng = np.random.default_rng(w * 7 + half)
    parts, sizes = [flat(rng, w, 40, half) for _ in range(320)], [(w, 40)] * 320
    ops, paths, n = pack_batch(parts, sizes)
    for rule in (_abi.NONZERO, _abi.EVENODD):
        want, got = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
        oracle.fill_batch(0, rule, ops, paths, 0, want, n_threads=8)
        fill_batch(ctx, ops, paths, 0, got, rule)
        assert_same(got, want, f"{w} {half} {rule}")


@pytest.mark.parametrize("w,h", [(5, 900), (300, 70), (1000, 900), (1031, 1030), (4099, 300)])
@pytest.mark.parametrize("half", [3000, 16000])
def test_flat_segments_single(ctx, w, h, half):
    rng = np.random.default_rng(w + half)
    for fmt in (_abi.MATTE8, _abi.RGBA8P):
        got, want, *_ = gpu_vs_oracle(ctx, flat(rng, w, h, half), w, h, fmt=fmt, clr=(9, 8, 7, 99), init=37)
        assert_same(got, want, f"{w}x{h}")
