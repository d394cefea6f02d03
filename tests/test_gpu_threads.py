"""One context per host thread: calls on small and on large canvases side by side.  The kernels'
limit of dynamic shared memory belongs to the device, so no thread's call may take it from
another's between that one's set-up and launch."""
import threading

import numpy as np
import pytest

import oracle
from footile_gb300 import _abi, workloads
from footile_gb300._lib import Context
from footile_gb300.path import FillRule
from footile_gb300.plotter import Plotter, fill_batch, pack_batch

pytestmark = pytest.mark.gpu


def _jobs():
    """Two jobs (a closure and what it must give) per kernel family, of small and of large bands."""
    rng = np.random.default_rng(11)
    out = []
    for w, h in ((40, 33), (900, 700), (1200, 1000), (4096, 300)):  # tile rasteriser, single bands
        ops = workloads.random_path(rng, min(w, h), 20)
        want = np.zeros((h, w), np.uint8)
        oracle.fill(_abi.NONZERO, ops, want, _abi.MATTE8)

        def job(ctx, ops=ops, shape=(h, w)):
            return Plotter(np.zeros(shape, np.uint8), context=ctx).fill(FillRule.NonZero, ops)
        out.append((job, want))
    for n, side in ((3, 48), (3, 1100), (400, 32)):
        parts = [workloads.random_path(rng, side, 12) for _ in range(n)]
        ops, paths, nbytes = pack_batch(parts, [side] * n)
        for stroke in (False, True):
            want = np.zeros(nbytes, np.uint8)
            oracle.fill_batch(int(stroke), 0, ops, paths, 0, want, n_threads=4)

            def job(ctx, ops=ops, paths=paths, nbytes=nbytes, stroke=stroke):
                got = np.zeros(nbytes, np.uint8)
                fill_batch(ctx, ops, paths, 0, got, 0, stroke)
                return got
            out.append((job, want))
    return out


def test_threads_do_not_take_each_others_shared_memory(cuda_ok, gpu_lib):
    jobs, errors, gate = _jobs(), [], threading.Barrier(3)

    def work(k):
        try:
            ctx = Context(0)
            order = np.random.default_rng(k)
            gate.wait(60)
            for _ in range(150):
                job, want = jobs[int(order.integers(len(jobs)))]
                if not np.array_equal(job(ctx), want):
                    raise AssertionError("wrong bytes")
            ctx.close()
        except Exception as e:  # noqa: BLE001 — reported by the test
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors, errors
