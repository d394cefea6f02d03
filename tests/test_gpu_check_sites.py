"""The bounds-check build's checks are reached, and pass, in every kernel that draws: the tile
rasteriser's two shapes (row ranges, batches; rows written in place, as whole lines of host
memory and through the staged bytes), the single-call bands, the CTA builds and the ordered
compositor with a pool full to its last edge, the coverage adjoint."""
import os
import subprocess
import sys
import textwrap

import pytest

from footile_gb300 import _build

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = textwrap.dedent("""
    import ctypes, sys
    import numpy as np, torch
    sys.path.insert(0, ROOT); sys.path.insert(0, ROOT + "/tests")
    from footile_gb300 import _abi, _lib, workloads
    L = _lib.load(path=LIB)
    import oracle
    from footile_gb300._lib import Context
    from footile_gb300.adjoint import Adjoint, pack_coverage
    from footile_gb300.plotter import fill_batch, composite_batch, pack_batch
    from helpers import gpu_vs_oracle
    ctx, rng = Context(0), np.random.default_rng(3)

    def reached():
        v = ctypes.c_ulonglong()
        assert L.ft_check_reached(ctypes.byref(v)) == 0
        return {k for k in range(64) if v.value >> k & 1}

    def clean(what, *sites):
        site = ctypes.c_int32(-1)
        assert L.ft_check_failures(ctypes.byref(site), None) == 0
        assert site.value == 0, (what, site.value)
        got = reached()
        assert set(sites) <= got, (what, sites, got)

    def single(w, h, stroke=False, **kw):
        ops = workloads.random_path(rng, max(w, h), 60, n_sub=2)
        init = rng.integers(0, 256, (h, w, 4) if kw.get("fmt") else (h, w)).astype(np.uint8)
        got, want, *_ = gpu_vs_oracle(ctx, ops, w, h, init=init, stroke=stroke, **kw)
        assert np.array_equal(got, want), (w, h, stroke, kw)

    def batch(sides, fmt=0, pinned=False, rule=0):
        ops, paths, n = pack_batch([workloads.random_path(rng, s, 12) for s in sides], sides, fmt,
                                   rng.integers(0, 256, (len(sides), 4)))
        if pinned:  # rows without padding: whole lines leave
            paths["stride"] = paths["width"]
            size = paths["stride"].astype(np.int64) * paths["height"]
            paths["raster_offset"], n = np.cumsum(size) - size, int(size.sum())
        want = np.zeros(n, np.uint8)
        oracle.fill_batch(0, rule, ops, paths, fmt, want, n_threads=8)
        keep = torch.zeros(n, dtype=torch.uint8)
        keep = keep.pin_memory() if pinned else keep
        pin = torch.from_numpy(ops.view(np.uint8)).pin_memory()
        got = keep.numpy()
        fill_batch(ctx, pin.numpy().view(_abi.OP_DTYPE) if pinned else ops, paths, fmt, got, rule)
        assert np.array_equal(got, want), (sides, fmt, pinned)

    reached()
    for w, h in ((256, 256), (97, 61), (900, 700)):
        single(w, h)
        single(w, h, fmt=_abi.RGBA8P, clr=(9, 8, 7, 99))
    clean("row ranges", 18, 19, 20, 21, 22, 23, 25)
    sides = [int(s) for s in rng.integers(1, 300, 400)]
    batch(sides)
    clean("batch", 18, 19, 20, 21, 22, 23, 25)
    batch(sides, pinned=True, rule=1)
    clean("batch into host rows", 18, 24, 25)
    batch(sides, fmt=_abi.RGBA8P)
    clean("batch in colour", 18, 24, 25)
    for w, h in ((1031, 1030), (4096, 300)):
        for stroke in (False, True):
            single(w, h, stroke)
            single(w, h, stroke, fmt=_abi.RGBA8P, clr=(9, 8, 7, 99))
    clean("bands", 18, 19, 26, 27, 28)

    # the ordered compositor: the smallest pool that the edges fit (one launch fewer than with a rerun)
    n, w, h = 40, 1000, 120
    parts = [workloads.random_path(rng, 1.0, 12) for _ in range(n)]
    for k, o in enumerate(parts):  # each call in a part of the row: empty bins in the others
        o["v"][:, 0::2] = o["v"][:, 0::2] * 200 + (k % 5) * 200
        o["v"][:, 1::2] *= h
    ops, paths, _ = pack_batch(parts, [(w, h)] * n, _abi.RGBA8P, rng.integers(0, 100, (n, 4)) + [0, 0, 0, 100])
    want = np.zeros((h, w, 4), np.uint8)
    oracle.composite(0, 0, ops, paths, _abi.RGBA8P, want)

    def launches(pool, tile_w):
        ctx.tune(pool_edges=pool, tile_w=tile_w)
        got, before = np.zeros((h, w, 4), np.uint8), ctx.launch_count()
        composite_batch(ctx, ops, paths, _abi.RGBA8P, got)
        assert np.array_equal(got, want), pool
        return ctx.launch_count() - before

    for tile_w in (256, 512, 1024):
        fewest = launches(1 << 20, tile_w)
        lo, hi = 1, 1 << 20
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (mid, hi) if launches(mid, tile_w) > fewest else (lo, mid)
        launches(hi, tile_w)
        clean("pool of %d edges" % hi, 6, 7, 8, 9, 10, 11, 17)
    ctx.set_tuning(None)

    ops, paths, n = pack_coverage([workloads.random_path(rng, 64, 10) for _ in range(20)], [64] * 20)
    adj = Adjoint(ctx)
    cov = np.zeros(n // 4, np.float32)
    for stroke in (False, True):
        adj.forward(0, ops, paths, cov, stroke)
        adj.backward(np.ones_like(cov), np.zeros((len(ops), 6), np.float32))
    adj.close()
    clean("adjoint", 30, 31)
    ctx.close()
    print("all sites clean")
""")


def test_checks_are_reached_and_pass(cuda_ok, tmp_path):
    lib = _build.build_variant(str(tmp_path / "check"), ["-DFT_CHECK=1"])
    code = f"ROOT = {ROOT!r}\nLIB = {lib!r}\n" + CASES
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=900, cwd=ROOT)
    assert out.returncode == 0 and "all sites clean" in out.stdout, out.stdout[-2000:] + out.stderr[-3000:]
