"""The adjoint's two lists (hits, then lit rays) and its chunks of thetas: views of odd
sizes whose rays cross warps and blocks, a view without a hit, every number of formula
parameters from none to four, both dual precisions."""

import math

import numpy as np
import pytest
import torch

from numericdream_b200 import abi, runtime, workloads

pytestmark = pytest.mark.gpu


def _setup(ctx, sides):
    views, cams = [], []
    for i, (w, h) in enumerate(sides):
        v, cam = workloads.mandelbulb_512(runtime.find_formula, power=8.0 - 0.6 * i, yaw=0.3 * i, pitch=0.1)
        if i == 1:  # looks away: no hits
            v.fwd[:] = [-x for x in v.fwd]
        v.width, v.height, v.tile_w, v.tile_h = w, h, w, h
        views.append(v)
        cams.append(cam)
    n = workloads.rays(views)
    g = runtime.GBuffer.allocate(n)
    ctx.forward(views, g)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    w = torch.rand(n, generator=gen, device="cuda") - 0.5
    w[::7] = 0.0  # rays without a weight
    return views, cams, g, w


@pytest.mark.parametrize("sides", [[(1, 1)], [(37, 29), (16, 8), (61, 17)], [(129, 65), (1, 1), (33, 31)]])
@pytest.mark.parametrize("precision", [32, 64])
def test_gradient_is_the_weighted_sum_of_the_jacobian(ctx, sides, precision):
    views, cams, g, w = _setup(ctx, sides)
    full = None
    for idx in ((0, 1, 2, 3), (0, 2), (2, 0, 1), (0,), ()):
        grad, per = ctx.backward(views, cams, g, w, param_idx=idx, de_precision=precision, per_ray=True)
        alone = ctx.backward(views, cams, g, w, param_idx=idx, de_precision=precision)
        k = len(idx) + 3
        off = 0
        for i, v in enumerate(views):
            n = workloads.rays([v])
            rows = (per[off:off + n] * w[off:off + n, None].double())
            want, size = rows.sum(0), rows.abs().sum(0)
            # sums of n doubles in two orders differ by at most n ulps of their sizes
            tol = size * n * np.finfo(np.float64).eps + 1e-300
            assert bool(((grad[i] - want).abs() <= tol).all()) and bool(((alone[i] - want).abs() <= tol).all())
            off += n
        miss = g.normal[:, 3] < 0.5
        assert not bool(per[miss].any())
        assert per.shape[1] == k
        if full is None:
            full = (idx, per)
            continue
        # a theta's column does not depend on which others are asked for: exactly so in FP32
        # (one theta to an evaluation); FP64 chunks hold other neighbours, same arithmetic
        cols = [full[0].index(p) for p in idx] + [4, 5, 6]
        ref = full[1][:, cols]
        if precision == 32:
            assert torch.equal(per, ref)
        else:
            assert bool(((per - ref).abs() <= 1e-9 * ref.abs().max(0).values.clamp_min(1e-30)).all())
    assert math.isfinite(float(full[1].abs().sum()))
