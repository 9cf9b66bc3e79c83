"""atan2 and pow of the FP32 DE on the device (branch-free special cases, nd_wgsl.h): a
formula that returns them, registered at run time, at points of every special case."""

import numpy as np
import pytest

from numericdream_b200 import abi, runtime

pytestmark = pytest.mark.gpu

SOURCE = """// @param Which min=0 max=1 default=0
fn de_iterations(p: Params) -> i32 { return 1; }
fn de_step(carry: IterCarry, pos: vec3f, p: Params) -> IterCarry {
    return IterCarry(vec3f(select(atan2(pos.y, pos.x), pow(pos.x, pos.z), p[0] > 0.5), 0.0, 0.0), 1.0);
}
fn de_finalize(carry: IterCarry) -> f32 { return carry.z.x; }
"""


@pytest.fixture(scope="module")
def formula(ndlib):
    return runtime.register_formula(SOURCE)


def _values(ctx, formula, which, pts):
    v = abi.make_view(formula, 8, 8, (0, 0, -3.0), params=[float(which)])
    return ctx.de_points(v, np.asarray(pts, np.float64), de_precision=32)[0]


def test_atan2(ctx, formula):
    inf, nan, tiny = np.inf, np.nan, 1e-30
    special = [0.0, -0.0, 1.0, -1.0, tiny, -tiny, 3e37, -3e37, inf, -inf, nan]
    yx = [(y, x) for y in special for x in special]
    rng = np.random.default_rng(2)
    yx += list(rng.normal(size=(4000, 2)) * 10.0 ** rng.uniform(-30, 30, (4000, 1)))
    got = _values(ctx, formula, 0, [(x, y, 0.0) for y, x in yx])
    y, x = np.float32([a for a, _ in yx]).astype(np.float64), np.float32([b for _, b in yx]).astype(np.float64)
    want = np.arctan2(y, x)
    bad = np.isnan(x) | np.isnan(y)
    np.testing.assert_array_equal(np.isnan(got), bad)
    # the host bound of the polynomial (tests/test_wgsl_math.py), with 2.5 ulp more for the
    # quotient that f32 division may be off by
    assert np.abs(got - want)[~bad].max() <= 5e-7 + 2.5 * 2.0 ** -24
    equal = ~bad & (np.abs(x) == np.abs(y)) & (x != 0)
    assert np.abs(got - want)[equal].max() <= 5e-7
    zero = ~bad & (y == 0)
    np.testing.assert_array_equal(np.signbit(got[zero]), np.signbit(y[zero]))


def test_pow(ctx, formula):
    xs = [0.0, -0.0, 0.25, 1.0, 7.0, -1.0, -1e-3, -np.inf, np.nan]
    pts = [(x, 0.0, z) for x in xs for z in (1.0, 2.0, 7.5)]
    got = _values(ctx, formula, 1, pts)
    for (x, _, z), g in zip(pts, got):
        if np.isnan(x) or x < 0:
            assert np.isnan(g), (x, z, g)  # the base is never negative in WGSL; NaN here
        else:
            assert abs(g - abs(x) ** z) <= 2e-6 * abs(x) ** z, (x, z, g)
