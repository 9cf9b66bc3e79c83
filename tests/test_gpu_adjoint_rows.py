"""The adjoint's per-ray rows, entry by entry: against rows recorded from the library that
ran the whole adjoint of a ray in one lane, and over calls large enough that the kernels
stride over their lists and take the rays in more than one pass."""

import json
import os

import numpy as np
import pytest
import torch

from numericdream_b200 import runtime, workloads

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "adjoint_rows.json")


@pytest.mark.parametrize("precision", [32, 64])
def test_rows_keep_the_rounding_of_one_tangent_an_evaluation(ctx, precision):
    """A grazing ray multiplies an evaluation's rounding by 1e9 and more, so that another
    choice of fused products shows in single entries.  With the evaluations' bits kept, what
    may differ is the arithmetic after them: the norm of D, three divisions, two products of
    three terms, some 20 roundings of terms of the row's size; 64 are allowed."""
    with open(GOLDEN) as f:
        gold = json.load(f)
    vc = [workloads.mandelbulb_512(runtime.find_formula, size=gold["size"], **v) for v in gold["views"]]
    views, cams = [v for v, _ in vc], [c for _, c in vc]
    g = runtime.GBuffer.allocate(workloads.rays(views))
    ctx.forward(views, g, runtime.make_opts(de_precision=precision))
    _, per = ctx.backward(views, cams, g, torch.ones_like(g.shade), param_idx=gold["param_idx"],
                          de_precision=precision, per_ray=True)
    per = per.cpu().numpy()
    want = np.zeros_like(per)
    for i, row in gold["rows"][str(precision)].items():
        want[int(i)] = row
    lit = (want != 0).any(1)
    assert lit.sum() > 200 and np.array_equal((per != 0).any(1), lit)
    size = np.maximum(np.abs(want[lit]), np.abs(want[lit]).max(1, keepdims=True))
    assert (np.abs(per[lit] - want[lit]) <= 64 * np.finfo(np.float64).eps * size).all()


def _problem(ctx, sides, precision):
    vc = [workloads.mandelbulb_512(runtime.find_formula, power=8.0 - 0.7 * i, yaw=0.4 * i, pitch=0.1)
          for i in range(len(sides))]
    views, cams = [v for v, _ in vc], [c for _, c in vc]
    for v, (w, h) in zip(views, sides):
        v.width, v.height, v.tile_w, v.tile_h = w, h, w, h
    n = workloads.rays(views)
    g = runtime.GBuffer.allocate(n)
    ctx.forward(views, g, runtime.make_opts(de_precision=precision))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    return views, cams, g, torch.rand(n, generator=gen, device="cuda") - 0.5


# lanes that take several items (a resident grid is at most 148 x 8 blocks of 128 lanes, the
# items are the lit rays times the thetas), views that change between a lane's items
STRIDED = [(331, 257), (129, 65), (1, 1), (517, 389), (97, 211)]
# more rays than one pass works on (2^22), the last pass ragged, a view across both
PASSES = [(1531, 1201), (1, 1), (1777, 1361)]


@pytest.mark.parametrize("sides,idx,precision", [
    (STRIDED, (0, 1, 2, 3), 32), (STRIDED, (0, 1, 2, 3), 64), (STRIDED, (0, 2), 32), (STRIDED, (), 64),
    (PASSES, (0, 2), 32), (PASSES, (0,), 64)])
def test_strides_and_passes_cover_every_ray_once(ctx, sides, idx, precision):
    views, cams, g, w = _problem(ctx, sides, precision)
    total = workloads.rays(views)
    if sides is PASSES:
        assert (1 << 22) < total
    grad, per = ctx.backward(views, cams, g, w, param_idx=idx, de_precision=precision, per_ray=True)
    lit = (per != 0).any(1)
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 128
    assert int(lit.sum()) * per.shape[1] > lanes
    off = 0
    for i, v in enumerate(views):
        n = workloads.rays([v])
        # the view by itself: other lists, another pass, the same rows
        one = runtime.GBuffer.allocate(n)
        for name in ("normal", "depth64", "shade"):
            getattr(one, name).copy_(getattr(g, name)[off:off + n])
        _, rows = ctx.backward([v], [cams[i]], one, w[off:off + n].contiguous(), param_idx=idx,
                               de_precision=precision, per_ray=True)
        assert torch.equal(rows, per[off:off + n])
        part = per[off:off + n] * w[off:off + n, None].double()
        want, size = part.sum(0), part.abs().sum(0)
        # sums of n doubles in two orders differ by at most n ulps of their sizes
        assert bool(((grad[i] - want).abs() <= size * n * np.finfo(np.float64).eps + 1e-300).all())
        off += n


def test_a_ray_beside_the_polar_axis_has_finite_derivatives(ctx):
    """x^2 + y^2 is subnormal there and its reciprocal infinite: atan2's tangent has to
    divide by it, or the ray's NaN is its whole view's gradient."""
    v, cam = workloads.mandelbulb_512(runtime.find_formula, size=1)
    v.cam_pos[0] = 1e-160
    g = runtime.GBuffer.allocate(1)
    ctx.forward([v], g, runtime.make_opts(de_precision=64))
    grad, per = ctx.backward([v], [cam], g, torch.ones_like(g.shade), param_idx=(0, 2), de_precision=64, per_ray=True)
    assert bool((per != 0).any()) and bool(torch.isfinite(per).all()) and bool(torch.isfinite(grad).all())
