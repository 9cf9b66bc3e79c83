"""The adjoint's per-ray rows, entry by entry, against rows recorded from the library that
ran the whole adjoint of a ray in one lane; and a ray beside the polar axis."""

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


def test_a_ray_beside_the_polar_axis_has_finite_derivatives(ctx):
    """x^2 + y^2 is subnormal there and its reciprocal infinite: atan2's tangent has to
    divide by it, or the ray's NaN is its whole view's gradient."""
    v, cam = workloads.mandelbulb_512(runtime.find_formula, size=1)
    v.cam_pos[0] = 1e-160
    g = runtime.GBuffer.allocate(1)
    ctx.forward([v], g, runtime.make_opts(de_precision=64))
    grad, per = ctx.backward([v], [cam], g, torch.ones_like(g.shade), param_idx=(0, 2), de_precision=64, per_ray=True)
    assert bool((per != 0).any()) and bool(torch.isfinite(per).all()) and bool(torch.isfinite(grad).all())
