"""Float SrcOver and its adjoint against the recurrence in 64 bits, where the kernels differ: fewer
layers than a step, steps and layers left over, canvases on either side of the rounds
that the shapes of the forward and of the backward fill."""
import numpy as np
import pytest

from footile_gb300.adjoint import srcover_backward, srcover_forward

pytestmark = pytest.mark.gpu


def reference(cov, clr, init, g):
    cov, clr, c = cov.astype(np.float64), clr.astype(np.float64), init.astype(np.float64)
    before = []
    for v, k in zip(cov, clr):
        before.append(c)
        c = k * v[:, None] + c * (1 - k[3] * v)[:, None]
    P, gcov = np.ones(cov.shape[1]), np.empty_like(cov)
    for n in range(len(cov) - 1, -1, -1):
        gcov[n] = P * ((g * clr[n]).sum(1) - clr[n][3] * (g * before[n]).sum(1))
        P = P * (1 - clr[n][3] * cov[n])
    return c, gcov, g * P[:, None]


@pytest.mark.parametrize("n_px", [1, 127, 128, 129, 12 * 128, "8", "9", "12", "16"])
@pytest.mark.parametrize("n", [1, 3, 4, 7, 8, 9, 16, 19])
def test_sizes(ctx, n, n_px):
    import torch

    if isinstance(n_px, str):  # one pixel into that many CTAs per SM
        n_px = int(n_px) * torch.cuda.get_device_properties(0).multi_processor_count * 128 + 1
    rng = np.random.default_rng(n)
    cov = np.where(rng.random((n, n_px)) < 0.3, rng.random((n, n_px)), rng.integers(0, 2, (n, n_px))).astype(np.float32)
    clr, init, g = (rng.random(s).astype(np.float32) for s in ((n, 4), (n_px, 4), (n_px, 4)))
    t = lambda a: torch.from_numpy(a).cuda()
    out, gcov, ginit = torch.empty(n_px, 4).cuda(), torch.empty(n, n_px).cuda(), torch.empty(n_px, 4).cuda()
    srcover_forward(ctx, t(cov.ravel()), n, n_px, t(clr), out, init=t(init))
    srcover_backward(ctx, t(cov.ravel()), n, n_px, t(clr), t(g), gcov, init=t(init), grad_init=ginit)
    want = reference(cov, clr, init, g)
    # a layer rounds five times; values up to 1 (the canvas), 4 (a gradient's dot product)
    eps = np.finfo(np.float32).eps
    for got, ref, top in zip((out, gcov, ginit), want, (1, 4, 1)):
        assert np.abs(got.cpu().numpy() - ref).max() <= top * 5 * (n + 2) * eps
