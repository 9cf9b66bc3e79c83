"""The watchdog reaches the bisections that the march leaves to the surface pass: a budget of
thousands of exact FP64 bisections on rays that march in a few probes."""

import ctypes as C

import pytest
import torch

from numericdream_b200 import abi, runtime, workloads

pytestmark = pytest.mark.gpu


def _view(budget):
    # a coarse eps seen from close by: some ten probes of microseconds each, then a chain of
    # 4096 bisections a ray
    return abi.make_view(runtime.find_formula("mandelbulb_bailout"), 48, 48, (0.0, 0.0, -2.2), params=[8.0, 6.0, 2.0],
                         max_steps=64, eps_coef=1e-3, eps_floor=0.0, refine_budget=budget,
                         flags=abi.ND_VIEW_EXACT_HIT)


def _run(ctx, budget, **kw):
    v = _view(budget)
    g = runtime.GBuffer.allocate(workloads.rays([v]))
    g.depth.fill_(float("nan"))
    ctx.forward([v], g, runtime.make_opts(kernel=abi.ND_KERNEL_PERSISTENT, de_precision=64, **kw))
    st = abi.nd_stats()
    status = ctx.lib.nd_last_stats(ctx.handle, C.byref(st))
    return status, st, g


def test_a_long_bisection_is_stopped_and_reported(ctx):
    _run(ctx, 4096)  # the kernels are loaded at their first launch
    status, full, before = _run(ctx, 4096)
    n = before.depth.numel()
    assert status == abi.ND_OK and full.rays == n and full.hits > 100 and full.timeouts == 0
    took = full.march_ms + full.shade_ms
    assert took > 8.0
    status, st, cut = _run(ctx, 4096, watchdog_ms=1)
    assert status == abi.ND_ERR_TIMEOUT and st.timeouts > 0
    assert st.march_ms + st.shade_ms < 0.6 * took and st.rays < n
    # what was not finished is not written
    assert int(torch.isnan(cut.depth).sum()) == n - st.rays
    # a budget of ordinary size is not touched by it, and the context goes on
    status, st, _ = _run(ctx, 40, watchdog_ms=1)
    assert status == abi.ND_OK and st.rays == n
    status, st, after = _run(ctx, 4096)
    assert status == abi.ND_OK and st.timeouts == 0
    for name in ("depth", "depth64", "steps", "evals", "normal"):
        assert torch.equal(getattr(before, name), getattr(after, name)), name
