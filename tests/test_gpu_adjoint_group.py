"""The adjoint of a batch that one formula group covers (one lane per listed ray): the
gradient is the weighted sum of the Jacobian, over views of odd sizes, a view without a hit,
rays without a weight and a list longer than the resident grid."""

import numpy as np
import pytest
import torch

from numericdream_b200 import abi, runtime, workloads

pytestmark = pytest.mark.gpu

GROUP = ((workloads.MANDELBULB, [8.0, 8.0], 2.6), (workloads.MANDELBOX, workloads.mandelbox_params(), 4.6),
         (workloads.MENGER, workloads.menger_params(), 2.6))


@pytest.mark.parametrize("sides", [[(37, 29), (16, 8), (61, 17)], [(613, 517), (701, 433), (129, 65)]])
@pytest.mark.parametrize("precision", [32, 64])
def test_gradient_is_the_weighted_sum_of_the_jacobian(ctx, sides, precision):
    if not {n for n, _, _ in GROUP} <= set(runtime.formula_names()):
        pytest.skip("the build has not the group's formulas")
    views, cams = [], []
    for i, ((w, h), (name, params, dist)) in enumerate(zip(sides, GROUP)):
        cam = abi.orbit_camera(yaw=0.3 * i, pitch=0.2, dist=dist, fov_y_deg=60.0)
        v = abi.make_view(runtime.find_formula(name), w, h, (0.0, 0.0, -dist), params=params, eps_coef=1e-4, eps_floor=0.0,
                          refine_budget=40, flags=abi.ND_VIEW_EXACT_HIT, light_dir=list(workloads.LIGHT_DIR),
                          normal_mode=abi.ND_NORMAL_CENTRAL, normal_h_coef=1e-4)
        runtime.orbit_view(cam, v)
        views.append(v)
        cams.append(cam)
    views[2].fwd[:] = [-x for x in views[2].fwd]  # looks away: no hits
    n = workloads.rays(views)
    g = runtime.GBuffer.allocate(n)
    ctx.forward(views, g, runtime.make_opts(de_precision=precision))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    w = torch.rand(n, generator=gen, device="cuda") - 0.5
    w[::7] = 0.0
    grad, per = ctx.backward(views, cams, g, w, param_idx=(0, 1), de_precision=precision, per_ray=True)
    assert int((per != 0).any(1).sum()) > 100 and not bool(per[g.normal[:, 3] < 0.5].any())
    off = 0
    for i, v in enumerate(views):
        k = workloads.rays([v])
        rows = per[off:off + k] * w[off:off + k, None].double()
        # sums of k doubles in two orders differ by at most k ulps of their sizes
        tol = rows.abs().sum(0) * k * np.finfo(np.float64).eps + 1e-300
        assert bool(((grad[i] - rows.sum(0)).abs() <= tol).all())
        off += k
    assert not bool(grad[2].any())
