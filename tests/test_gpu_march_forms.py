"""The deferred march (probes in the march, bisection in the surface pass) against the
plain launch, which runs march_to's loop inline: every G-buffer output bit for bit, over
the forms of the march (bisection budgets, exact hits, verified steps, high quality,
normal modes, shadows), the edges of its limits, odd sizes and both DE precisions."""

import pytest
import torch

from numericdream_b200 import abi, runtime, workloads

pytestmark = pytest.mark.gpu

FORMS = {
    "bisect4": {},
    "bisect0": {"refine_budget": 0},
    "bisect1": {"refine_budget": 1},
    "exact1": {"refine_budget": 1, "flags": abi.ND_VIEW_EXACT_HIT},
    "exact40": {"refine_budget": 40, "flags": abi.ND_VIEW_EXACT_HIT, "eps_coef": 1e-4, "eps_floor": 0.0},
    "verify20hq": {"refine_budget": 20, "march_verify": 1, "high_quality": 1},
    "verify0": {"refine_budget": 0, "march_verify": 1},
    "central_shadow": {"normal_mode": abi.ND_NORMAL_CENTRAL, "shadow": 1, "light_dir": list(workloads.LIGHT_DIR)},
    "steps0": {"max_steps": 0},
    "steps0_exact": {"max_steps": 0, "flags": abi.ND_VIEW_EXACT_HIT},
    "steps0_bisect1": {"max_steps": 0, "refine_budget": 1},
    "steps0_none": {"max_steps": 0, "refine_budget": 0},
    "steps1": {"max_steps": 1},
    "steps7": {"max_steps": 7, "eps_coef": 5e-2},
    "far": {"max_dist": 2.2},
    "safety": {"step_safety": 0.6, "max_steps": 40},
}


def _view(form, w, h, spp=1, inside=False):
    # `inside`: the camera sits where the first sample is below eps
    pos = (0.0, 0.0, -0.2) if inside else (0.6, 0.5, -2.2)
    return abi.make_view(runtime.find_formula("mandelbulb_bailout"), w, h, pos, params=[7.0, 9.0, 2.0], spp=spp, seed=9,
                         **FORMS[form])


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("precision", [32, 64])
def test_deferred_march_equals_the_plain_launch(ctx, form, precision):
    for views in ([_view(form, 53, 37)], [_view(form, 40, 31, 2), _view(form, 1, 1), _view(form, 33, 9, 1, True)]):
        n = workloads.rays(views)
        out, counts = [], []
        for kernel in (abi.ND_KERNEL_PLAIN, abi.ND_KERNEL_PERSISTENT):
            g = runtime.GBuffer.allocate(n)
            for t in (g.depth, g.normal, g.trap, g.shade, g.shadow, g.depth64):
                t.fill_(float("nan"))
            ctx.forward(views, g, runtime.make_opts(kernel=kernel, de_precision=precision))
            st = ctx.stats()
            counts.append((st.rays, st.hits, st.march_evals, st.normal_evals, st.shadow_evals))
            out.append(g)
        for name in ("depth", "normal", "trap", "steps", "iters", "shade", "shadow", "depth64", "evals"):
            a, b = getattr(out[0], name), getattr(out[1], name)
            assert torch.equal(a, b), f"{name}: {(a != b).sum().item()} values differ"
        assert counts[0] == counts[1]


def test_lite_and_shadows_of_one_view_equal_those_in_a_batch(ctx):
    """One view's constants travel in kernel parameters, a batch's in memory: the same bits."""
    views = [_view("central_shadow", 61, 43), _view("central_shadow", 17, 9, 2)]
    lite = abi.make_lite([((0.1, 0.2, 0.3), 0.0, 0.4, 1.4), ((0.9, 0.5, 0.2), 1.0, 0.7, 1.6)],
                         [(abi.ND_LIGHT_GLOBAL, (0.4, 0.8, -0.45), (1.0, 0.9, 0.8), 1.1)])

    def outputs(vs):
        g = runtime.GBuffer.allocate(workloads.rays(vs))
        ctx.forward(vs, g, runtime.make_opts(kernel=abi.ND_KERNEL_PERSISTENT))
        return torch.cat([ctx.shade_lite(vs, [lite] * len(vs), g), g.shadow[:, None], g.shade[:, None]], 1)

    assert torch.equal(outputs(views), torch.cat([outputs([v]) for v in views]))


@pytest.mark.parametrize("w,h,spp", [(191, 97, 1), (130, 127, 1), (16391, 1, 1), (1, 16384, 1), (3, 5462, 2), (65, 127, 2),
                                     (128, 128, 1)])
def test_plain_launch_in_blocks_marches_every_ray(ctx, w, h, spp):
    """Views large enough for the plain launch's 8 x 4 blocks: tiles that no block fits, and
    remainders on both sides."""
    v = _view("bisect4", w, h, spp)
    n = workloads.rays([v])
    out = []
    for kernel in (abi.ND_KERNEL_PLAIN, abi.ND_KERNEL_PERSISTENT):
        g = runtime.GBuffer.allocate(n)
        g.steps.fill_(-1)
        ctx.forward([v], g, runtime.make_opts(kernel=kernel))
        assert ctx.stats().rays == n
        out.append(g)
    for name in ("depth", "normal", "trap", "steps", "evals"):
        assert torch.equal(getattr(out[0], name), getattr(out[1], name)), name
